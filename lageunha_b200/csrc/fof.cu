// Friends-of-friends groups on the engine's sorted particles and octree.
//
// Reference: pnew_fof_link (FoF/fof.c:217-290) grows a group from a seed,
// linking every particle whose distance to a member is <= fof_link, which
// PreFoF (Cosmos/PreFoF.c:267-385) runs cell by cell with a linking length
// FOF_LINK = 0.2 mean separations and keeps groups of at least FOF_MINNUM =
// 20 members. The groups are the connected components of the "distance <=
// link" relation, so any linking order gives the same partition. Here every
// warp of sorted particles searches the 4-cell cubes within the link, down the
// octree of the force evaluation, and joins the linked particles in a lock-free
// union-find; the roots then count their members, and
// every particle of a group of >= min_members gets the group's smallest
// caller index as its label (-1 otherwise).
#include <math.h>

#include "ctx.cuh"
#include "short_range.cuh"

using namespace tpm;

namespace {

// Nodes a warp holds. 32 are taken at a time while their children, eight each,
// leave room for what single ones may still add: a node taken alone adds at most
// 7 on each level below a cube, of which the smallest mesh (16 cells, 2 levels of
// cubes) has most. So no set of particles can overflow it. 544 entries are the
// most before a wide step.
constexpr int kFofDeep = 7 * (kAxisBits - 2), kFofWide = 7 * 32;
constexpr int kFofStack = 544 + kFofWide + kFofDeep;
constexpr int kFofThreads = 128;
// A warp's particles of one cube are split by octants while their smallest common
// cube reaches kFofFar particles past them and is wider than kFofKeep links (see
// k_fof_link)
constexpr int kFofFar = 128;
constexpr float kFofKeep = 2.f;
static_assert(kFofStack * sizeof(uint32_t) * (kFofThreads / 32) * 16 <= 227 * 1024, "16 blocks per SM");

TPM_D uint32_t find_root(uint32_t *parent, uint32_t x) {
  uint32_t p = parent[x];
  while (p != x) {
    uint32_t g = parent[p];
    parent[x] = g;  // path halving; racing writers only shorten paths
    x = p;
    p = g;
  }
  return x;
}

TPM_D void unite(uint32_t *parent, uint32_t a, uint32_t b) {
  while (true) {
    a = find_root(parent, a);
    b = find_root(parent, b);
    if (a == b) return;
    if (a > b) {
      uint32_t t = a;
      a = b;
      b = t;
    }
    // hook the larger root under the smaller one, if it is still a root
    uint32_t old = atomicCAS(&parent[b], b, a);
    if (old == b) return;
    b = old;
  }
}

__global__ void k_fof_init(uint32_t *parent, uint32_t *gsize, uint32_t *label, int64_t np) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x) {
    parent[i] = (uint32_t)i;
    gsize[i] = 0;
    label[i] = 0xffffffffu;
  }
}

// A warp takes 32 consecutive sorted particles, those of one 4-cell cube at a
// time, so that its lanes share one search: the cubes within the link of their
// box, from each cube's tree node down (nodes beyond the link of the box
// pruned, 32 classified at a time), and the particles of the leaves found are
// tested by all lanes. A node whose cube's diagonal is within the link is a
// clique: each of its particles joins the node's first one, and a particle
// outside needs only one link into it, and none if both are in one group
// already, which spares a dense clump nearly all of its pairs. Nodes that lie
// wholly before the particles are left out: a pair is found from its first
// particle's side.
//
// In a dense cube 32 consecutive particles may lie on both sides of an octant's
// face, their box many times as large as either part's, so those are searched for
// one after the other: a cube of 128 particles and more besides is dense enough,
// and one wider than two links, since the link widens the box of each part as well.
// 60 thousand particles of a Gaussian clump (0.5 cells, link 0.05): 2.06 -> 0.41 ms,
// half a million in a tighter one 13.3 -> 1.15 ms, the clustered 160^3 field at link
// 0.2 3.65 -> 2.79 ms (all with labels in device memory); 64, 256 and 512 particles,
// 0.5 and 1 links: within 10%, or twice as long at links of a cell.
//
// One thread per particle ran with 2.7 of 32 lanes active (each had its own
// stack and met its leaves at its own time): 8.4 ms for the 4.1 million
// particles of the clustered 160^3 field.
__global__ void __launch_bounds__(kFofThreads) k_fof_link(const uint32_t *__restrict__ spos,
                                                          const uint64_t *__restrict__ skey, int cube_shift,
                                                          int keep_shift,
                                                          const uint4 *__restrict__ walkA,
                                                          const uint4 *__restrict__ walkB,
                                                          const uint32_t *__restrict__ cube_node,
                                                          const uint32_t *__restrict__ start_cube, int64_t np, int n,
                                                          float cpu, float link, float clique_half, uint32_t *parent,
                                                          uint32_t *err) {
  __shared__ uint32_t stacks[kFofThreads / 32][kFofStack];
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t *stack = stacks[threadIdx.x >> 5];
  const float link2 = link * link, near2 = link2 * 1.0001f + 1e-12f;
  // the cubes' faces lie a float rounding of a coordinate away at most
  const float reach = link * 1.001f + 1e-3f;
  const int64_t step = (int64_t)gridDim.x * kFofThreads;
  for (int64_t base = (blockIdx.x * (int64_t)kFofThreads + threadIdx.x) - lane; base < np; base += step) {
    const int64_t i64 = base + lane;
    const uint32_t i = (uint32_t)i64;
    const bool valid = i64 < np;
    uint32_t p[3] = {0, 0, 0};
    uint64_t key = 0;
    if (valid) {
      p[0] = spos[3 * i64 + 0];
      p[1] = spos[3 * i64 + 1];
      p[2] = spos[3 * i64 + 2];
      key = skey[i64];
    }
    uint32_t root = i;  // a root of this particle at some time
    unsigned rest = __ballot_sync(0xffffffffu, valid);
    while (rest) {
      const int lead = __ffs(rest) - 1;
      const uint64_t k0 = __shfl_sync(0xffffffffu, key, lead);
      unsigned members = __ballot_sync(0xffffffffu, valid && key >> cube_shift == k0 >> cube_shift) & rest;
      while (true) {
        const int last = 31 - __clz(members);
        const uint64_t differ = k0 ^ __shfl_sync(0xffffffffu, key, last);
        if (!differ) break;
        const int shift = 3 * ((63 - __clzll((long long)differ)) / 3 + 1);  // of the smallest cube with all of them
        if (shift <= keep_shift) break;
        const int64_t before = base + lead - kFofFar, after = base + last + kFofFar;
        if (!(before >= 0 && skey[before] >> shift == k0 >> shift) && !(after < np && skey[after] >> shift == k0 >> shift))
          break;
        members &= __ballot_sync(0xffffffffu, key >> (shift - 3) == k0 >> (shift - 3));
      }
      rest &= ~members;
      const bool mine = (members >> lane) & 1u;
      const uint32_t first = (uint32_t)(base + lead);
      // the members' box: its middle (fixed point and cells) and half sizes
      float half[3], at[3];
      uint32_t mid[3];
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const uint32_t ref = __shfl_sync(0xffffffffu, p[a], lead);
        float x = mine ? wrapf(p[a], ref, cpu) : 0.f, lo = x, hi = x;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
          hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        half[a] = 0.5f * (hi - lo);
        at[a] = __uint2float_rn(ref) * cpu + 0.5f * (lo + hi);
        mid[a] = ref + (uint32_t)__float2int_rn(0.5f * (lo + hi) / cpu);
      }
      // joins the members to the particles of [s, e) that are linked to them
      auto join = [&](uint32_t s, uint32_t e, bool clique, bool near) {
        bool need = mine;
        if (clique) {
          need = mine && near;
          if (mine && i >= s && i < e) {
            if (i > s) unite(parent, i, s);
            need = false;
          }
          if (!__any_sync(0xffffffffu, need)) return;
          const uint32_t rs = __shfl_sync(0xffffffffu, lane == 0 ? find_root(parent, s) : 0u, 0);
          if (need && root != rs) root = find_root(parent, i);
          need = need && root != rs;
          if (!__any_sync(0xffffffffu, need)) return;
        }
        for (uint32_t j0 = s; j0 < e; j0 += 32) {
          const int m = (int)min(32u, e - j0);
          uint32_t q[3] = {0, 0, 0};
          if (lane < m)
            for (int a = 0; a < 3; a++) q[a] = spos[3 * (int64_t)(j0 + lane) + a];
          for (int k = 0; k < m; k++) {
            float ex = wrapf(__shfl_sync(0xffffffffu, q[0], k), p[0], cpu);
            float ey = wrapf(__shfl_sync(0xffffffffu, q[1], k), p[1], cpu);
            float ez = wrapf(__shfl_sync(0xffffffffu, q[2], k), p[2], cpu);
            const uint32_t j = j0 + k;
            if (need && (clique || j > i) && ex * ex + ey * ey + ez * ez <= link2) {
              unite(parent, i, j);
              if (clique) need = false;
            }
            __syncwarp();
          }
          if (clique && !__any_sync(0xffffffffu, need)) return;
        }
      };
      int run[3][4], ntot[3], stotal = 1;
#pragma unroll
      for (int a = 0; a < 3; a++) {
        axis_runs(at[a] - half[a] - reach, at[a] + half[a] + reach, n, run[a]);
        ntot[a] = run[a][1] + run[a][3];
        stotal *= ntot[a];
      }
      for (int jb = 0; jb < stotal; jb += 32) {
        const int j = jb + lane;
        uint32_t node = kNoNode, s = 0, e = 0;
        if (j < stotal) {
          const int jj[3] = {j % ntot[0], (j / ntot[0]) % ntot[1], j / (ntot[0] * ntot[1])};
          uint32_t cc[3];
#pragma unroll
          for (int a = 0; a < 3; a++)  // the second run starts at cube 0
            cc[a] = (uint32_t)(jj[a] < run[a][1] ? run[a][0] + jj[a] : jj[a] - run[a][1]);
          const uint64_t id = morton3(cc[0], cc[1], cc[2]);
          node = cube_node[id];
          s = start_cube[id];
          e = start_cube[id + 1];
          if (e <= first) e = s;
        }
        // cubes without a node hold fewer than kLeafMin particles
        unsigned bare = __ballot_sync(0xffffffffu, node == kNoNode && e > s);
        while (bare) {
          const int k = __ffs(bare) - 1;
          bare &= bare - 1;
          join(__shfl_sync(0xffffffffu, s, k), __shfl_sync(0xffffffffu, e, k), false, true);
        }
        const unsigned nodes = __ballot_sync(0xffffffffu, node != kNoNode && e > s);
        if (node != kNoNode && e > s) stack[__popc(nodes & lt)] = node;
        int top = __popc(nodes);
        __syncwarp();
        while (top > 0) {
          const int take = min(top, top + kFofWide + kFofDeep <= kFofStack ? 32 : 1);
          const bool has = lane < take;
          uint4 rec = make_uint4(0, 0, 0, 0), geo = rec;
          if (has) {
            const uint32_t nd = stack[top - take + lane];
            rec = walkB[nd];
            geo = walkA[2 * (int64_t)nd];
          }
          __syncwarp();
          top -= take;
          const float nh = __uint_as_float(geo.w);
          const bool clique = nh <= clique_half;
          int kind = 0;  // 1: open, 2: join
          const uint32_t nch = rec.w & 0xffffu;
          if (has && rec.x + rec.y > first) {
            // the image nearest to the middle of the box has the smallest gap to
            // it (the one nearest to a member at its edge may be on the far side)
            float dx = fmaxf(fabsf(wrapf(geo.x, mid[0], cpu)) - nh - half[0], 0.f);
            float dy = fmaxf(fabsf(wrapf(geo.y, mid[1], cpu)) - nh - half[1], 0.f);
            float dz = fmaxf(fabsf(wrapf(geo.z, mid[2], cpu)) - nh - half[2], 0.f);
            // the box's own rounding beside the pair's
            if (dx * dx + dy * dy + dz * dz <= near2 + 1e-6f) kind = nch == 0 || (clique && rec.y <= 32u) ? 2 : 1;
          }
          // children of the opened nodes
          uint32_t incl = kind == 1 ? nch : 0u;
          const uint32_t push = incl;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
          }
          const int total = (int)__shfl_sync(0xffffffffu, incl, 31);
          if (top + total > kFofStack) {
            if (lane == 0) atomicOr(err, (uint32_t)kErrStackOverflow);
            top = 0;
            break;
          }
          for (uint32_t k = 0; k < push; k++) stack[top + (int)(incl - push + k)] = rec.z + k;
          top += total;
          __syncwarp();
          unsigned found = __ballot_sync(0xffffffffu, kind == 2);
          while (found) {
            const int k = __ffs(found) - 1;
            found &= found - 1;
            const uint32_t s2 = __shfl_sync(0xffffffffu, rec.x, k), c2 = __shfl_sync(0xffffffffu, rec.y, k);
            const bool cl = __shfl_sync(0xffffffffu, (int)clique, k);
            bool near = true;
            if (cl) {
              const float h2 = __shfl_sync(0xffffffffu, nh, k);
              float dx = fmaxf(fabsf(wrapf(__shfl_sync(0xffffffffu, geo.x, k), p[0], cpu)) - h2, 0.f);
              float dy = fmaxf(fabsf(wrapf(__shfl_sync(0xffffffffu, geo.y, k), p[1], cpu)) - h2, 0.f);
              float dz = fmaxf(fabsf(wrapf(__shfl_sync(0xffffffffu, geo.z, k), p[2], cpu)) - h2, 0.f);
              near = dx * dx + dy * dy + dz * dz <= near2;
            }
            join(s2, s2 + c2, cl, near);
          }
        }
      }
    }
  }
}

// After the links: every particle's root, found without rewriting parent (a
// path-splitting write racing with another thread's could leave an entry on
// an inner node), and the member count of every root.
__global__ void k_fof_count(const uint32_t *__restrict__ parent, uint32_t *root, uint32_t *gsize, int64_t np) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t x = (uint32_t)i, p = parent[x];
    while (p != x) {
      x = p;
      p = parent[x];
    }
    root[i] = x;
    atomicAdd(&gsize[x], 1u);
  }
}

__global__ void k_fof_label_min(const uint32_t *root, const uint32_t *gsize, const uint32_t *perm, int64_t np,
                                uint32_t min_members, uint32_t *label, uint32_t *ngroups) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t r = root[i];
    if (gsize[r] >= min_members) {
      atomicMin(&label[r], perm[i]);
      if (r == (uint32_t)i) atomicAdd(ngroups, 1u);
    }
  }
}

__global__ void k_fof_scatter(const uint32_t *root, const uint32_t *gsize, const uint32_t *perm, int64_t np,
                              uint32_t min_members, const uint32_t *label, int32_t *out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t r = root[i];
    out[perm[i]] = gsize[r] >= min_members ? (int32_t)label[r] : -1;
  }
}

int grid_of(int64_t n) {
  int64_t b = (n + 255) / 256;
  if (b > 148 * 16) b = 148 * 16;
  return (int)(b < 1 ? 1 : b);
}

}  // namespace

extern "C" {

int tpm_fof(tpm_ctx *c, float link, int32_t min_members, int32_t *labels, int mem, int64_t *ngroups) {
  if (!c || !labels || !(link > 0.f) || min_members < 1) return fail(TPM_E_ARG, "bad arguments to tpm_fof");
  if (c->np <= 0) return fail(TPM_E_STATE, "no particles loaded");
  if (2.f * link >= (float)c->prm.n_mesh) return fail(TPM_E_ARG, "link too large for the box");
  CK(cudaSetDevice(c->device));
  cudaStream_t st = c->st;
  int64_t np = c->np;
  // the sort and the octree of a force evaluation (no walk)
  int rc = enqueue_forces(c, TPM_PART_TREE, st, false, false);
  if (rc) return rc;
  // five words per particle, reusing the caller-order force scratch and the
  // alternate sort buffers, which hold nothing between evaluations
  uint32_t *parent = c->val_alt == c->perm ? c->val : c->val_alt;
  uint32_t *gsize = reinterpret_cast<uint32_t *>(c->key_alt == c->skey ? c->key : c->key_alt);
  uint32_t *label = gsize + np;
  int32_t *out = reinterpret_cast<int32_t *>(c->fout);
  uint32_t *root = reinterpret_cast<uint32_t *>(c->fout) + np;
  uint32_t *ng = c->tb.counters + kCntFofGroups;
  k_fof_init<<<grid_of(np), 256, 0, st>>>(parent, gsize, label, np);
  int lb = (int)((np + kFofThreads - 1) / kFofThreads);
  if (lb > 148 * 32) lb = 148 * 32;
  float cpu = (float)((double)c->g.n / 4294967296.0);
  // half side of the largest cube with a diagonal within the link
  const float clique_half = 0.999f * link / (2.f * sqrtf(3.f));
  // the bits per axis of the widest cube that is not split
  int keep = 0;
  while (keep < c->g.sub_bits + 2 && ldexpf(1.f, keep + 1 - c->g.sub_bits) <= kFofKeep * link) keep++;
  k_fof_link<<<lb, kFofThreads, 0, st>>>(c->spos, c->skey, 3 * (c->g.sub_bits + 2), 3 * keep, c->tb.walkA, c->tb.walkB,
                                         c->tb.cube_node, c->tb.start_cube, np, c->g.n, cpu, link, clique_half, parent,
                                         c->err);
  k_fof_count<<<grid_of(np), 256, 0, st>>>(parent, root, gsize, np);
  k_fof_label_min<<<grid_of(np), 256, 0, st>>>(root, gsize, c->perm, np, (uint32_t)min_members, label, ng);
  k_fof_scatter<<<grid_of(np), 256, 0, st>>>(root, gsize, c->perm, np, (uint32_t)min_members, label, out);
  CK(cudaGetLastError());
  uint32_t herr = 0, hng = 0;
  CK(cudaMemcpyAsync(&herr, c->err, sizeof(herr), cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(&hng, ng, sizeof(hng), cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(labels, out, sizeof(int32_t) * np,
                     mem == TPM_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  // the scratch buffers were overwritten: no forces are held
  c->parts_valid = 0;
  if (herr) return fail(herr & kErrStackOverflow ? TPM_E_OVERFLOW : TPM_E_CUDA, "device error flags 0x%x", herr);
  if (ngroups) *ngroups = hng;
  return 0;
}

}  // extern "C"
