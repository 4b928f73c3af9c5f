// Short-range force of ordinary density by direct summation (sm_100a).
//
// Inside the law's cut (rsphere, a few cells) the tree hardly accepts a node
// where there is about one particle per cell: the walk of the reference
// (OST/ost.ver2.c:247-306) then amounts to finding the particles in reach and
// summing over them, and finding them node by node, once per warp, costs more
// instructions than the pairs. Here a team of four warps takes the targets of
// one 4-cell cube. Each warp collects a quarter of the particles in the cube's
// reach, once, as floats relative to the cube's first target in shared memory,
// and evaluates that quarter against every target of the cube; the four
// partial forces are added in a fixed order, so the result does not depend on
// the scheduling. Cubes with more than kDirCandidates particles in the cubes
// around them (dense clumps, where the tree's nodes pay) are left to the tree
// walk as groups of its list.
//
// Per sub-group of at most 16 targets the warp drops the sources out of reach
// of the sub-group's own box and evaluates the rest, the half-warps taking
// alternate sources for the same targets: a box of 16 targets (about 4 x 2 x 2
// cells) has a fifth less reach volume than one of 32, which is what bounds
// the sum: three quarters of the evaluated pairs lie beyond the cut.
//
// Bound by the shared-memory pipe (75% busy at 128^3: the law table's gather,
// 3.2 wavefronts for a warp's pair step, and the source rows, 1.5), then by
// issue (62%). Short-range force of the 512^3 benchmark: 83.9 -> 78.3 ms against
// the walk, at 68.6 instead of 82.4 thousand million pairs and no node terms.
#include <algorithm>

#include "short_range.cuh"

namespace tpm {

constexpr int kDirTeams = 5;       // teams per CTA, one CTA per SM
constexpr int kDirWarps = 4;       // warps of a team
constexpr int kDirTeamThreads = 32 * kDirWarps;
constexpr int kDirThreads = kDirTeams * kDirTeamThreads;
constexpr int kDirSub = 16;        // targets per sub-group
constexpr int kDirTargets = 128;   // targets per pass over a cube's sources
constexpr int kDirCap = 416;       // sources a warp holds at a time
constexpr int kDirSeg = kDirCap + 64;   // padded to a multiple of 64
constexpr int kDirList = 192;      // sources evaluated per flush
constexpr int kDirRow = kDirList + 8;
// most particles in the cubes in reach: twice the mean of one per cell. Above
// it the tree's accepted nodes are the cheaper (clustered 256^3 field, direct
// sum and walk together: 20.2 ms at 3000, 21.6 at 4000, 23.5 at 6000, 20.7 all
// by the walk); below it the direct sum is (128^3 of the strongly displaced
// field with the 4-cell cut, one step: 3.20 ms at 3000, 3.09 at 4000, 3.47 all
// by the walk)
constexpr uint32_t kDirCandidates = 3500;
constexpr float kDirFar = -1.0e4f;  // a (negated) coordinate outside every cut

struct alignas(16) DirWarp {
  float seg[3][kDirSeg];   // the warp's share of the sources in reach, negated
  float list[3][kDirRow];  // those in reach of the current sub-group
  WalkBox box;             // the box of the current unit
};

struct DirTeam {
  float part[kDirWarps][3 * kDirTargets];  // the warps' partial forces
  float tgt[3][kDirTargets];
  float4 sbox[kDirTargets / kDirSub][2];   // sub-group boxes: centre, half sizes
  uint32_t next[2];                        // the team's coming unit
};

TPM_D void team_sync(int team) { asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(kDirTeamThreads) : "memory"); }

// The m sources of the list (padded here to a multiple of 8 with ones far
// outside the cut) against the lanes' targets, half-warp h taking the quads
// 2i + h.
template <bool kHardCut>
TPM_D void direct_eval(DirWarp &dw, int m, int lane, float ftx, float fty, float ftz, float rs2, uint32_t kcut,
                       uint32_t tlb, float2 a[6]) {
  const int m8 = (m + 7) & ~7;
  if (lane < m8 - m) {
    dw.list[0][m + lane] = kDirFar;
    dw.list[1][m + lane] = kDirFar;
    dw.list[2][m + lane] = kDirFar;
  }
  __syncwarp();
  const float2 tx = make_float2(ftx, ftx), ty = make_float2(fty, fty), tz = make_float2(ftz, ftz);
  const float *lx = dw.list[0] + (lane >> 4) * 4;
#pragma unroll 2
  for (int q = 0; q < m8; q += 8) {
    float4 x = *reinterpret_cast<const float4 *>(lx + q);
    float4 y = *reinterpret_cast<const float4 *>(lx + kDirRow + q);
    float4 z = *reinterpret_cast<const float4 *>(lx + 2 * kDirRow + q);
    pp_two<kHardCut>(make_float2(x.x, x.y), make_float2(y.x, y.y), make_float2(z.x, z.y), tx, ty, tz, rs2, kcut, tlb,
                     a[0], a[1], a[2]);
    pp_two<kHardCut>(make_float2(x.z, x.w), make_float2(y.z, y.w), make_float2(z.z, z.w), tx, ty, tz, rs2, kcut, tlb,
                     a[3], a[4], a[5]);
  }
  __syncwarp();
}

template <bool kHardCut>
__global__ void __launch_bounds__(kDirThreads, 1)
    k_direct(const WalkBox *__restrict__ boxes, const uint32_t *__restrict__ uprefix, int nbox,
             uint32_t *__restrict__ unext, uint32_t *__restrict__ stats, const float2 *__restrict__ glog, float rsphere,
             uint32_t kcut) {
  extern __shared__ float4 smem4[];
  const float rs2 = rsphere * rsphere;
  float2 *tl = reinterpret_cast<float2 *>(smem4);
  DirTeam *teams = reinterpret_cast<DirTeam *>(smem4 + kLogSmemF4);
  DirWarp *warps = reinterpret_cast<DirWarp *>(teams + kDirTeams);
  const uint32_t nunits = nbox == 1 ? boxes[0].counters[kCntUnits] : uprefix[nbox];
  if (nunits == 0) return;
  for (int i = threadIdx.x; i <= kLogEntries; i += kDirThreads) tl[i] = glog[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int team = wib / kDirWarps, tw = wib % kDirWarps, ttid = threadIdx.x - team * kDirTeamThreads;
  DirTeam &T = teams[team];
  DirWarp &dw = warps[wib];
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t tlb = (uint32_t)__cvta_generic_to_shared(tl) - (uint32_t)(kLogBase * 8);
  // a little slack against float rounding of the relative coordinates
  const float prune = rs2 * 1.0001f + 1e-4f;
  // the reach tests use differences scaled by 2^-7, so that the part beyond a
  // box comes from one saturating multiply-add (a difference over 128 cells
  // counts as 128, out of every reach)
  constexpr float kSc = 1.f / 128.f;
  const float prune_sc = prune * kSc * kSc;
  uint32_t npp = 0, nsubs = 0;
  int cur_box = -1, par = 0;
  if (ttid == 0) T.next[0] = atomicAdd(unext, 1u);
  team_sync(team);
  uint32_t u = T.next[0];
  while (u < nunits) {
    int b = 0;
    if (nbox > 1) {
      int lo = 0, hi = nbox - 1;
      while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (uprefix[mid] <= u) lo = mid;
        else hi = mid - 1;
      }
      b = lo;
      u -= uprefix[b];
    }
    if (b != cur_box) {
      const uint32_t *src = reinterpret_cast<const uint32_t *>(&boxes[b]);
      constexpr int kWords = (int)(sizeof(WalkBox) / 4);
      static_assert(kWords <= 32, "box record larger than a warp's load");
      uint32_t v = lane < kWords ? src[lane] : 0u;
      __syncwarp();
      if (lane < kWords) reinterpret_cast<uint32_t *>(&dw.box)[lane] = v;
      __syncwarp();
      cur_box = b;
    }
    const uint32_t cube = dw.box.units[u];
    const uint32_t s = dw.box.start_cube[cube];
    const int cnt = (int)(dw.box.start_cube[cube + 1] - s);
    const int n = dw.box.n_cells;
    const float cpu = dw.box.cpu;
    const float inv_n = __frcp_rn((float)n);
    // the cube: cells [c0, c0 + w) per axis (the last cube of a mesh that is no
    // multiple of four is narrower); coordinates are relative to its first
    // target, so that close pairs keep their small separations. Lane a works
    // out axis a: the cube's middle in cells and relative to that target, its
    // half width, and the runs of cubes in reach
    float mid[3], hw[3], ctr[3];
    uint32_t ref[3];
    int run0[3], nrun[3], ntot[3];
    {
      const int a = lane < 3 ? lane : 0;
      const int c0 = 4 * (int)compact3(cube >> a), w = min(4, n - c0);
      const uint32_t ur = dw.box.spos[3 * (int64_t)s + a];
      const uint64_t pr = (uint64_t)ur * (uint64_t)n;  // the target in cells, 32.32
      const float h = 0.5f * (float)w;
      const float off = (float)((int)(pr >> 32) - c0) + (float)(uint32_t)pr * 2.3283064365386963e-10f;
      const float reach = rsphere * kCubeReach;
      int run[4];
      axis_runs((float)c0 - reach, (float)(c0 + w) + reach, n, run);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        mid[k] = __shfl_sync(0xffffffffu, (float)c0 + h, k);
        hw[k] = __shfl_sync(0xffffffffu, h, k);
        ctr[k] = __shfl_sync(0xffffffffu, h - off, k);
        ref[k] = __shfl_sync(0xffffffffu, ur, k);
        run0[k] = __shfl_sync(0xffffffffu, run[0], k);
        nrun[k] = __shfl_sync(0xffffffffu, run[1], k);
        ntot[k] = __shfl_sync(0xffffffffu, run[1] + run[3], k);
      }
    }
    const int stotal = ntot[0] * ntot[1] * ntot[2];
    // the particle range of the j-th cube in reach (empty beyond the reach)
    const float inv_nx = __frcp_rn((float)ntot[0]), inv_ny = __frcp_rn((float)ntot[1]);
    auto cube_range = [&](int j, uint32_t &s0, uint32_t &c) {
      s0 = 0;
      c = 0;
      if (j >= stotal) return;
      // j = jx + nx (jy + ny jz): quotients exact from float reciprocals below
      // 2^20 cubes ((q + 0.5) / d lies 0.5 / d from an integer)
      int jj[3];
      if (stotal < (1 << 20)) {
        int qx = (int)(((float)j + 0.5f) * inv_nx);
        int qy = (int)(((float)qx + 0.5f) * inv_ny);
        jj[0] = j - qx * ntot[0];
        jj[1] = qx - qy * ntot[1];
        jj[2] = qy;
      } else {
        jj[0] = j % ntot[0];
        jj[1] = (j / ntot[0]) % ntot[1];
        jj[2] = j / (ntot[0] * ntot[1]);
      }
      uint32_t cc[3];
      float d2 = 0.f;
#pragma unroll
      for (int a = 0; a < 3; a++) {
        // the second run starts at cube 0
        const int c4 = jj[a] < nrun[a] ? run0[a] + jj[a] : jj[a] - nrun[a];
        cc[a] = (uint32_t)c4;
        const float e = cube_gap(c4, mid[a], hw[a], n, inv_n);
        d2 += e * e;
      }
      if (d2 < rs2) {
        uint32_t cid = (uint32_t)morton3(cc[0], cc[1], cc[2]);
        s0 = dw.box.start_cube[cid];
        c = dw.box.start_cube[cid + 1] - s0;
      }
    };
    uint32_t s0, c;
    for (int t0 = 0; t0 < cnt; t0 += kDirTargets) {
      const int tc = min(cnt - t0, kDirTargets);
      const int nsub = (tc + kDirSub - 1) / kDirSub, per = (tc + nsub - 1) / nsub;
      // targets and sub-group boxes: half-warp h of warp w takes sub-group 2 w + h
      {
        const int sub = 2 * tw + (lane >> 4), l16 = lane & 15, first = sub * per;
        const bool on = sub < nsub && l16 < min(per, tc - first);
        float lo[3] = {1e30f, 1e30f, 1e30f}, hi[3] = {-1e30f, -1e30f, -1e30f};
        if (on) {
          const uint32_t *p = dw.box.spos + 3 * (int64_t)(s + t0 + first + l16);
#pragma unroll
          for (int a = 0; a < 3; a++) {
            lo[a] = hi[a] = wrapf(p[a], ref[a], cpu);
            T.tgt[a][first + l16] = lo[a];
          }
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
          for (int a = 0; a < 3; a++) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
          }
        if (on && l16 == 0) {
          T.sbox[sub][0] = make_float4(0.5f * (lo[0] + hi[0]), 0.5f * (lo[1] + hi[1]), 0.5f * (lo[2] + hi[2]),
                                       -0.5f * (hi[0] - lo[0]) * kSc);
          T.sbox[sub][1] = make_float4(-0.5f * (hi[1] - lo[1]) * kSc, -0.5f * (hi[2] - lo[2]) * kSc, 0.f, 0.f);
        }
      }
      // the coming unit: read by the team after this pass's barriers, the slot
      // written again only after the next unit's
      const bool last = t0 + kDirTargets >= cnt;
      if (ttid == 0 && last) T.next[par ^ 1] = atomicAdd(unext, 1u);
      team_sync(team);
      if (tw == 0) nsubs += (uint32_t)nsub;
      bool first = true;
      for (int jb = 0; jb < stotal; jb += 32) {
        // the batch's particles as one range of flat indices; this warp takes
        // every fourth chunk of 32
        cube_range(jb + lane, s0, c);
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        const uint32_t batch = __shfl_sync(0xffffffffu, incl, 31);
        const uint32_t base = s0 - (incl - c);
        uint32_t v[3] = {0, 0, 0};
        auto load = [&](uint32_t t) {
          // the cube of flat index t: the number of cubes that end at or before it
          int L = 0;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            uint32_t e = __shfl_sync(0xffffffffu, incl, L + o - 1);
            if (e <= t) L += o;
          }
          const uint32_t i = t + __shfl_sync(0xffffffffu, base, L);
          if (t < batch) {
            const uint32_t *q = dw.box.spos + 3 * (int64_t)i;
            v[0] = q[0];
            v[1] = q[1];
            v[2] = q[2];
          }
        };
        uint32_t f = 32u * (uint32_t)tw;
        if (f < batch) load(f + lane);
        while (f < batch || (first && jb + 32 >= stotal)) {
          int seg = 0;
          while (f < batch && seg + 32 <= kDirCap) {
            const bool valid = f + lane < batch;
            const float px = wrapf(v[0], ref[0], cpu), py = wrapf(v[1], ref[1], cpu), pz = wrapf(v[2], ref[2], cpu);
            f += kDirTeamThreads;
            if (f < batch) load(f + lane);
            const float dx = fmaxf(fabsf(px - ctr[0]) - hw[0], 0.f), dy = fmaxf(fabsf(py - ctr[1]) - hw[1], 0.f),
                        dz = fmaxf(fabsf(pz - ctr[2]) - hw[2], 0.f);
            const bool keep = valid && dx * dx + dy * dy + dz * dz <= prune;
            const unsigned mk = __ballot_sync(0xffffffffu, keep);
            if (keep) {
              float *at = dw.seg[0] + seg + __popc(mk & lt);
              at[0] = -px;
              at[kDirSeg] = -py;
              at[2 * kDirSeg] = -pz;
            }
            seg += __popc(mk);
          }
          // pad to a multiple of 64
          dw.seg[0][seg + lane] = kDirFar;
          dw.seg[0][seg + 32 + lane] = kDirFar;
          __syncwarp();
          // every sub-group of targets against these sources
          for (int i = 0; i < nsub; i++) {
            const float4 b0 = T.sbox[i][0], b1 = T.sbox[i][1];
            const int t = i * per + (lane & 15);
            const bool act = (lane & 15) < min(per, tc - i * per);
            const float tx = act ? T.tgt[0][t] : b0.x, ty = act ? T.tgt[1][t] : b0.y, tz = act ? T.tgt[2][t] : b0.z;
            const float2 cx = make_float2(b0.x, b0.x), cy = make_float2(b0.y, b0.y), cz = make_float2(b0.z, b0.z);
            float2 a[6];
#pragma unroll
            for (int k = 0; k < 6; k++) a[k] = make_float2(0.f, 0.f);
            int len = 0;
            uint32_t kept = 0;
            for (int k0 = 0; k0 < seg; k0 += 64) {
              const float *sp = dw.seg[0] + k0 + 2 * lane;
              const float2 nx = *reinterpret_cast<const float2 *>(sp);
              const float2 ny = *reinterpret_cast<const float2 *>(sp + kDirSeg);
              const float2 nz = *reinterpret_cast<const float2 *>(sp + 2 * kDirSeg);
              // |n + c| = |p - c|: the sources are negated
              const float2 ex = __fadd2_rn(nx, cx), ey = __fadd2_rn(ny, cy), ez = __fadd2_rn(nz, cz);
              const float2 dx = make_float2(__saturatef(fmaf(fabsf(ex.x), kSc, b0.w)), __saturatef(fmaf(fabsf(ex.y), kSc, b0.w)));
              const float2 dy = make_float2(__saturatef(fmaf(fabsf(ey.x), kSc, b1.x)), __saturatef(fmaf(fabsf(ey.y), kSc, b1.x)));
              const float2 dz = make_float2(__saturatef(fmaf(fabsf(ez.x), kSc, b1.y)), __saturatef(fmaf(fabsf(ez.y), kSc, b1.y)));
              const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
              const bool k0p = d2.x <= prune_sc, k1p = d2.y <= prune_sc;
              const unsigned m0 = __ballot_sync(0xffffffffu, k0p), m1 = __ballot_sync(0xffffffffu, k1p);
              float *at = dw.list[0] + len + __popc(m0 & lt) + __popc(m1 & lt);
              if (k0p) {
                at[0] = nx.x;
                at[kDirRow] = ny.x;
                at[2 * kDirRow] = nz.x;
                at++;
              }
              if (k1p) {
                at[0] = nx.y;
                at[kDirRow] = ny.y;
                at[2 * kDirRow] = nz.y;
              }
              len += __popc(m0) + __popc(m1);
              if (len > kDirList - 64 || k0 + 64 >= seg) {
                direct_eval<kHardCut>(dw, len, lane, tx, ty, tz, rs2, kcut, tlb, a);
                kept += (uint32_t)len;
                len = 0;
              }
            }
            float fx = (a[0].x + a[0].y) + (a[3].x + a[3].y);
            float fy = (a[1].x + a[1].y) + (a[4].x + a[4].y);
            float fz = (a[2].x + a[2].y) + (a[5].x + a[5].y);
            fx += __shfl_xor_sync(0xffffffffu, fx, 16);
            fy += __shfl_xor_sync(0xffffffffu, fy, 16);
            fz += __shfl_xor_sync(0xffffffffu, fz, 16);
            if (act && lane < 16) {
              float *o = &T.part[tw][3 * t];
              if (!first) {
                fx += o[0];
                fy += o[1];
                fz += o[2];
              }
              o[0] = fx;
              o[1] = fy;
              o[2] = fz;
              npp += kept;
            }
          }
          first = false;
        }
      }
      team_sync(team);
      {
        const float md = dw.box.mass * dw.box.inv_ll;
        float *out = dw.box.ftree + 3 * (int64_t)(s + t0);
        for (int e = ttid; e < 3 * tc; e += kDirTeamThreads)
          out[e] = ((T.part[0][e] + T.part[1][e]) + (T.part[2][e] + T.part[3][e])) * md;
      }
    }
    par ^= 1;
    u = T.next[par];
  }
  unsigned long long np64 = npp;
  for (int o = 16; o > 0; o >>= 1) np64 += __shfl_down_sync(0xffffffffu, np64, o);
  if (lane == 0) {
    atomicAdd(reinterpret_cast<unsigned long long *>(&stats[kCntPp]), np64);
    if (tw == 0) atomicAdd(&stats[kCntSubs], nsubs);
  }
}

// Every non-empty 4-cell cube, in about Morton order, to the direct summation
// (units) or, with more than kDirCandidates particles in the cubes in reach, to
// the tree walk as groups of at most group_max particles.
__global__ void __launch_bounds__(256) k_tree_units(const uint32_t *__restrict__ start_cube, int64_t ncubes, int n,
                                                    float rsphere, uint32_t group_max, uint32_t *__restrict__ units,
                                                    uint32_t *__restrict__ groups, uint32_t *__restrict__ counters) {
  const int lane = threadIdx.x & 31;
  const float rs2 = rsphere * rsphere, inv_n = __frcp_rn((float)n), reach = rsphere * kCubeReach;
  for (int64_t c0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); c0 < ncubes;
       c0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = c0 + lane;
    uint32_t s = 0, cnt = 0, total = 0;
    if (c < ncubes) {
      s = start_cube[c];
      cnt = start_cube[c + 1] - s;
    }
    if (cnt) {
      int run[3][4];
      float mid[3], hw[3];
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const int x = 4 * (int)compact3((uint32_t)c >> a), w = min(4, n - x);
        hw[a] = 0.5f * (float)w;
        mid[a] = (float)x + hw[a];
        axis_runs((float)x - reach, (float)(x + w) + reach, n, run[a]);
      }
      auto at = [&](int a, int j) { return j < run[a][1] ? run[a][0] + j : j - run[a][1]; };  // the second run starts at 0
      for (int jz = 0; jz < run[2][1] + run[2][3] && total <= kDirCandidates; jz++) {
        const int cz = at(2, jz);
        const float ez = cube_gap(cz, mid[2], hw[2], n, inv_n);
        for (int jy = 0; jy < run[1][1] + run[1][3]; jy++) {
          const int cy = at(1, jy);
          const float ey = cube_gap(cy, mid[1], hw[1], n, inv_n);
          for (int jx = 0; jx < run[0][1] + run[0][3]; jx++) {
            const int cx = at(0, jx);
            const float ex = cube_gap(cx, mid[0], hw[0], n, inv_n);
            if (ex * ex + ey * ey + ez * ez < rs2) {
              const int64_t id = (int64_t)morton3((uint32_t)cx, (uint32_t)cy, (uint32_t)cz);
              total += min(start_cube[id + 1] - start_cube[id], 1u << 24);
            }
          }
        }
      }
    }
    const bool dense = total > kDirCandidates;
    const unsigned m = __ballot_sync(0xffffffffu, cnt && !dense);
    if (m) {
      uint32_t first = 0;
      if (lane == 0) first = atomicAdd(&counters[kCntUnits], (uint32_t)__popc(m));
      first = __shfl_sync(0xffffffffu, first, 0);
      if (cnt && !dense) units[first + __popc(m & ((1u << lane) - 1u))] = (uint32_t)c;
    }
    if (cnt && dense) {
      const uint32_t ng = (cnt + group_max - 1) / group_max;
      const int64_t g0 = atomicAdd(&counters[kCntGroups], ng);
      for (uint32_t g = 0; g < ng; g++) {
        groups[2 * (g0 + g)] = s + g * group_max;
        groups[2 * (g0 + g) + 1] = min(group_max, cnt - g * group_max);
      }
    }
  }
}

void tree_units(const TreeParams &tp, TreeBuffers &tb, cudaStream_t st, int64_t *launches) {
  int blocks = (int)std::min<int64_t>((tb.ncubes4 + 255) / 256, 148 * 16);
  k_tree_units<<<blocks, 256, 0, st>>>(tb.start_cube, tb.ncubes4, (int)tp.n, tp.rsphere,
                                       (uint32_t)std::max(1, std::min(32, tp.group_max)), tb.units, tb.groups,
                                       tb.counters);
  if (launches) *launches += 1;
}

void launch_direct(const WalkBox *boxes, const uint32_t *uprefix, int nbox, int64_t max_units, uint32_t *unext,
                   uint32_t *stats, const LawTable &law, float rsphere, cudaStream_t st) {
  const size_t smem = sizeof(float4) * kLogSmemF4 + sizeof(DirTeam) * kDirTeams + sizeof(DirWarp) * kDirTeams * kDirWarps;
  static_assert(sizeof(DirTeam) % 16 == 0 && sizeof(DirWarp) % 16 == 0, "float4 alignment");
  static_assert(sizeof(float4) * kLogSmemF4 + sizeof(DirTeam) * kDirTeams + sizeof(DirWarp) * kDirTeams * kDirWarps <=
                    232448,
                "shared memory of one SM");
  // an attribute of the function on the current device, set on every launch
  // so that every device and thread has it
  cudaFuncSetAttribute(k_direct<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaFuncSetAttribute(k_direct<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // a block fills its SM, so blocks that would find no unit are left out: a
  // small box's PM chain runs beside the sum on the SMs that remain
  const int grid = (int)std::min<int64_t>(sms, (max_units + kDirTeams - 1) / kDirTeams);
  const float rs2 = rsphere * rsphere;
  const uint32_t kcut = law_cut_bin(law, rs2);
  if (law.hard_cut)
    k_direct<true><<<grid, kDirThreads, smem, st>>>(boxes, uprefix, nbox, unext, stats, law.tlog, rsphere, kcut);
  else
    k_direct<false><<<grid, kDirThreads, smem, st>>>(boxes, uprefix, nbox, unext, stats, law.tlog, rsphere, kcut);
}

}  // namespace tpm
