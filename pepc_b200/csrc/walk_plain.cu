// walk_plain.cu -- FP64 tree walks (the drop-in "plain" form) and the
// traversal orchestration of pepc_traverse_tree.
//
// Two semantics, both exact:
//  * per target (module_tree_walk_pthreads.f90:558-765): every target keeps
//    its own next-node index in the RPO node order; a warp of 32 key-ordered
//    targets processes, at each step, the smallest next index among its lanes
//    (all lanes that wait for that node evaluate it together, the node data is
//    loaded once).  Each lane sees exactly its own LIFO sequence, so its
//    interaction list, order and counts equal the reference's.
//  * per tile (module_tree_walk_simple.f90:256-384): a warp holds one tile of
//    <= 32 targets; a twig is opened if any target fails the MAC, children are
//    visited first to last (key order) through the fwd pointers.
// Compiled with --fmad=false: results are bit-identical to the oracle.

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "internal.cuh"

namespace pepcg {

namespace {

constexpr int kWalkThreads = 128;

struct WalkArgs {
  int64_t nt;
  const double* tx;
  const double* ty;
  const double* tz;
  const double4* nc4;
  const int2* meta;
  const int2* fwd;
  const double* mom;
  const int32_t* nleaves;
  const double* bl2;   // boxlength2[0..20]
  const double* macb;  // per-twig MAC threshold, or nullptr: bl2 of the level (Barnes-Hut)
  const double* tq;    // force_law 5: the targets' charges
  double kinv, sqrtpi;  // force_law 5: kelbg_invsqrttemp, sqrt(acos(-1))
  const double* vbox;  // 3 * nbox
  int nbox;
  double theta2, eps2;
  int32_t M;
  int64_t npart;
  double* ex;
  double* ey;
  double* ez;
  double* pot;
  double* work;
  unsigned long long* counters;  // [0] leaf, [1] twig, [2] mac
  uint32_t* status;
  unsigned int* queue;           // bucket counter, zeroed before the launch
  // per tile
  const int2* tiles;  // (first target, count)
  int64_t ntiles;
  // packed per-tile walk
  const int2* fwdf;     // (first child, next after the subtree) as forward-preorder indices
  const int32_t* tflag;  // per target: length of the tile starting there, else 0
  const int32_t* pstart;  // packed per-tile walk: first target of each pack, then nt
  const int32_t* npacks;  // the number of packs (device)
  // spatial_interaction_cutoff (module_mirror_boxes.f90:52), when finite
  int has_cut;
  double cut[3];
  // list walk (k_walk_list64)
  const LevelRecord* drec;
  const int32_t* rpo2fpo;
  const int32_t* fpo2rpo;
  uint2* lstack;       // kListStack entries per resident block
  int lper;            // per target: targets per bucket (8, 16 or 32)
  // what k_walk_list64 left to k_walk_target64 / k_walk_tilepack64 (kOnly): [0] their
  // number, then targets (count << 20 | first) or packs
  int32_t* over;
  const uint32_t* tree_status;  // set: drec was not built
};

// any(abs(delta) >= spatial_interaction_cutoff) (module_tree_walk_pthreads.f90:
// 622,639; module_tree_walk_simple.f90:330,377): the node is skipped.  The walks
// are instantiated with and without the test (kCut), so that a walk without a
// finite cutoff runs the code it ran before the option existed.
template <bool kCut>
__device__ __forceinline__ bool cut_off(const WalkArgs& A, double dx, double dy, double dz) {
  return kCut && (fabs(dx) >= A.cut[0] || fabs(dy) >= A.cut[1] || fabs(dz) >= A.cut[2]);
}

__device__ __forceinline__ void warp_add_counters(unsigned long long* ctr, unsigned long long a,
                                                  unsigned long long b, unsigned long long c) {
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&ctr[0], a);
    atomicAdd(&ctr[1], b);
    atomicAdd(&ctr[2], c);
  }
}

constexpr int kOverShift = 20;

// kOnly: walks the targets that A.over lists (a separate instantiation: the test inside
// the queue loop cost the walk of 250,000 targets 10 %)
template <int kLaw, bool kCut, bool kOnly = false>
__global__ void __launch_bounds__(kWalkThreads) k_walk_target64(WalkArgs A) {
  __shared__ double s_bl2[kMaxLevel + 1];
  __shared__ double s_vb[3 * 125];
  for (int i = threadIdx.x; i <= kMaxLevel; i += blockDim.x) s_bl2[i] = A.bl2[i];
  for (int i = threadIdx.x; i < 3 * A.nbox; i += blockDim.x) s_vb[i] = A.vbox[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const unsigned M = (unsigned)A.M;
  unsigned long long c_leaf = 0, c_twig = 0, c_mac = 0;
  for (;;) {
    unsigned b = 0;
    if (lane == 0) b = atomicAdd(A.queue, 1u);
    b = __shfl_sync(0xffffffffu, b, 0);
    int64_t t0 = (int64_t)b * 32;
    int per = 32;
    if constexpr (kOnly) {
      if ((int)b >= A.over[0]) break;
      const int o = A.over[1 + b];
      t0 = o & ((1 << kOverShift) - 1);
      per = o >> kOverShift;
    }
    if (t0 >= A.nt) break;
    const int64_t t = t0 + lane;
    const bool valid = t < A.nt && (!kOnly || lane < per);
    double px = 0, py = 0, pz = 0, e0 = 0, e1 = 0, e2 = 0, ph = 0, w = 0;
    KelbgArgs kel{0.0, A.kinv, A.sqrtpi};
    if (valid) {
      px = A.tx[t]; py = A.ty[t]; pz = A.tz[t];
      if (kLaw == 5) kel.tq = A.tq[t];
      e0 = A.ex[t]; e1 = A.ey[t]; e2 = A.ez[t]; ph = A.pot[t]; w = A.work[t];
    }
    bool complete = true;
    for (int ib = 0; ib < A.nbox; ++ib) {
      // shifted_particle_position = x - vbox (module_tree_walk_pthreads.f90:595)
      const double sx = px - s_vb[3 * ib], sy = py - s_vb[3 * ib + 1], sz = pz - s_vb[3 * ib + 2];
      // the root is never evaluated: the walk starts with its children (:601)
      unsigned next = valid ? 1u : M;
      int64_t partner = 0;
      for (;;) {
        const unsigned u = __reduce_min_sync(0xffffffffu, next);
        if (u >= M) break;
        if (next != u) continue;
        const double4 a = A.nc4[u];
        const int2 mu = A.meta[u];
        const double dx = sx - a.x, dy = sy - a.y, dz = sz - a.z;
        const double dist2 = (dx * dx + dy * dy) + dz * dz;
        if (mu.y & kLeafFlag) {
          partner += 1;
          w += 1.0;  // counted before the cutoff test (:620-622)
          if (!cut_off<kCut>(A, dx, dy, dz)) {
            ++c_leaf;
            if (dist2 > 0.0) {
              double fx, fy, fz, fp;
              law_leaf64<kLaw>(a.w, dx, dy, dz, dist2, A.eps2, fx, fy, fz, fp, kel);
              e0 += fx; e1 += fy; e2 += fz; ph += fp;
            }
          }
          next = u + 1;
        } else {
          ++c_mac;
          if (A.theta2 * dist2 > (A.macb ? A.macb[u] : s_bl2[mu.y & 0xff])) {
            partner += A.nleaves[u];
            if (!cut_off<kCut>(A, dx, dy, dz)) {
              double m[9];
#pragma unroll
              for (int k = 0; k < 9; ++k) m[k] = A.mom[kMomStride * (int64_t)u + k];
              double fx, fy, fz, fp;
              law_twig64<kLaw>(a.w, m, dx, dy, dz, dist2, A.eps2, fx, fy, fz, fp);
              e0 += fx; e1 += fy; e2 += fz; ph += fp;
              ++c_twig;
              w += 1.0;
            }
            next = (unsigned)mu.x;
          } else {
            next = u + 1;
          }
        }
      }
      if (valid && partner != A.npart) complete = false;
    }
    if (valid) {
      A.ex[t] = e0; A.ey[t] = e1; A.ez[t] = e2; A.pot[t] = ph; A.work[t] = w;
    }
    if (__any_sync(0xffffffffu, !complete) && lane == 0) atomicOr(A.status, ST_INCOMPLETE);
  }
  warp_add_counters(A.counters, c_leaf, c_twig, c_mac);
}

// One warp per tile (PER_TILE tiles of up to 32 targets) or per group-walk
// bucket (GROUP: kTPL x 32 key-consecutive targets, kTPL targets per lane,
// lane k holding targets t0 + k + 32 s).  A twig is accepted only if every
// target of the tile passes the MAC (module_tree_walk_simple.f90:343-382);
// children are visited first to last through fwd, so each target's
// interactions come in the reference's order.
// Launch bounds: six resident blocks per SM for one target per lane (the
// plain group walk at 4M takes 223 ms against 270 ms at the unbounded 108
// registers), four for two.
template <int kLaw, int kTPL, bool kCut>
__global__ void __launch_bounds__(kWalkThreads, kTPL == 1 ? 6 : 4) k_walk_tile64(WalkArgs A) {
  __shared__ double s_bl2[kMaxLevel + 1];
  __shared__ double s_vb[3 * 125];
  for (int i = threadIdx.x; i <= kMaxLevel; i += blockDim.x) s_bl2[i] = A.bl2[i];
  for (int i = threadIdx.x; i < 3 * A.nbox; i += blockDim.x) s_vb[i] = A.vbox[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const unsigned M = (unsigned)A.M;
  constexpr int kB = 32 * kTPL;  // GROUP bucket size
  unsigned long long c_leaf = 0, c_twig = 0, c_mac = 0;
  for (;;) {
    unsigned b = 0;
    if (lane == 0) b = atomicAdd(A.queue, 1u);
    b = __shfl_sync(0xffffffffu, b, 0);
    const int64_t nbk = A.tiles ? A.ntiles : (A.nt + kB - 1) / kB;
    if ((int64_t)b >= nbk) break;
    const int2 tl = A.tiles ? A.tiles[b]
                            : make_int2((int)((int64_t)b * kB), (int)min((int64_t)kB, A.nt - (int64_t)b * kB));
    bool valid[kTPL];
    int64_t t[kTPL];
    double px[kTPL], py[kTPL], pz[kTPL], e0[kTPL], e1[kTPL], e2[kTPL], ph[kTPL], w[kTPL];
    KelbgArgs kel[kTPL];
#pragma unroll
    for (int s = 0; s < kTPL; ++s) {
      valid[s] = lane + 32 * s < tl.y;
      t[s] = (int64_t)tl.x + lane + 32 * s;
      px[s] = py[s] = pz[s] = e0[s] = e1[s] = e2[s] = ph[s] = w[s] = 0.0;
      kel[s] = KelbgArgs{0.0, A.kinv, A.sqrtpi};
      if (valid[s]) {
        px[s] = A.tx[t[s]]; py[s] = A.ty[t[s]]; pz[s] = A.tz[t[s]];
        if (kLaw == 5) kel[s].tq = A.tq[t[s]];
        e0[s] = A.ex[t[s]]; e1[s] = A.ey[t[s]]; e2[s] = A.ez[t[s]]; ph[s] = A.pot[t[s]];
        w[s] = A.work[t[s]];
      }
    }
    bool complete = true;
    for (int ib = 0; ib < A.nbox; ++ib) {
      const double vx = s_vb[3 * ib], vy = s_vb[3 * ib + 1], vz = s_vb[3 * ib + 2];
      unsigned u = 0;  // tree_walk_single_aux starts at the root (:286)
      int64_t partner = 0;
      while (u < M) {
        const double4 a = A.nc4[u];
        const int2 mu = A.meta[u];
        const int2 fw = A.fwd[u];
        // d = (x - vbox) - coc (module_tree_walk_simple.f90:328,345)
        double dx[kTPL], dy[kTPL], dz[kTPL], dist2[kTPL];
#pragma unroll
        for (int s = 0; s < kTPL; ++s) {
          dx[s] = (px[s] - vx) - a.x; dy[s] = (py[s] - vy) - a.y; dz[s] = (pz[s] - vz) - a.z;
          dist2[s] = (dx[s] * dx[s] + dy[s] * dy[s]) + dz[s] * dz[s];
        }
        if (mu.y & kLeafFlag) {
          partner += 1;
#pragma unroll
          for (int s = 0; s < kTPL; ++s)
            if (valid[s] && !cut_off<kCut>(A, dx[s], dy[s], dz[s])) {
              w[s] += 1.0;
              ++c_leaf;
              if (dist2[s] > 0.0) {
                double fx, fy, fz, fp;
                law_leaf64<kLaw>(a.w, dx[s], dy[s], dz[s], dist2[s], A.eps2, fx, fy, fz, fp, kel[s]);
                e0[s] += fx; e1[s] += fy; e2[s] += fz; ph[s] += fp;
              }
            }
          u = (unsigned)fw.y;
        } else {
          const double thr = A.macb ? A.macb[u] : s_bl2[mu.y & 0xff];
          // MAC evaluations stop at the tile's first failing target, in
          // target order (:343-370)
          int first_fail = kB;
          unsigned any_fail = 0;
#pragma unroll
          for (int s = 0; s < kTPL; ++s) {
            const bool ok = !valid[s] || (A.theta2 * dist2[s] > thr);
            const unsigned fail = __ballot_sync(0xffffffffu, !ok);
            if (fail && first_fail == kB) first_fail = 32 * s + __ffs(fail) - 1;
            any_fail |= fail;
          }
#pragma unroll
          for (int s = 0; s < kTPL; ++s)
            if (valid[s] && lane + 32 * s <= first_fail) ++c_mac;
          if (any_fail == 0) {
            partner += A.nleaves[u];
            double m[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) m[k] = A.mom[kMomStride * (int64_t)u + k];
#pragma unroll
            for (int s = 0; s < kTPL; ++s)
              if (valid[s] && !cut_off<kCut>(A, dx[s], dy[s], dz[s])) {
                double fx, fy, fz, fp;
                law_twig64<kLaw>(a.w, m, dx[s], dy[s], dz[s], dist2[s], A.eps2, fx, fy, fz, fp);
                e0[s] += fx; e1[s] += fy; e2[s] += fz; ph[s] += fp;
                w[s] += 1.0;
                ++c_twig;
              }
            u = (unsigned)fw.y;
          } else {
            u = (unsigned)fw.x;
          }
        }
      }
      if (partner != A.npart) complete = false;
    }
#pragma unroll
    for (int s = 0; s < kTPL; ++s)
      if (valid[s]) {
        A.ex[t[s]] = e0[s]; A.ey[t[s]] = e1[s]; A.ez[t[s]] = e2[s]; A.pot[t[s]] = ph[s];
        A.work[t[s]] = w[s];
      }
    if (!complete && lane == 0) atomicOr(A.status, ST_INCOMPLETE);
  }
  warp_add_counters(A.counters, c_leaf, c_twig, c_mac);
}

// Tiles of the grown particles: tree nodes with <= T leaves whose parent has
// more than T (the key-prefix split of tree_walk_init_aux,
// module_tree_walk_simple.f90:168-211, is exactly this set of nodes).
// Several reference tiles per warp (simple-walk semantics, module_tree_walk_
// simple.f90:256-385).  Each warp takes one pack of consecutive whole tiles
// of at most 32 targets (k_pack_tiles).  Every tile walks the tree in forward
// preorder (children first to
// last); the warp steps through the union of its tiles' walks in that order:
// at each step the lanes whose tile stands at the smallest forward-preorder
// index f evaluate node f together (one load for all of them), and each tile
// decides accept / open by a ballot over its own lanes.  A lane's sequence of
// interactions is exactly its tile's, so fields, work and MAC counts equal
// the one-tile-per-warp walk's.
template <int kLaw, bool kCut, bool kOnly = false>
// Six resident blocks per SM (80 registers, a few spilled): at 4M, T = 16,
// 260 ms against 296 ms at the unbounded 110 registers (four blocks).
__global__ void __launch_bounds__(kWalkThreads, 6) k_walk_tilepack64(WalkArgs A) {
  __shared__ double s_bl2[kMaxLevel + 1];
  __shared__ double s_vb[3 * 125];
  for (int i = threadIdx.x; i <= kMaxLevel; i += blockDim.x) s_bl2[i] = A.bl2[i];
  for (int i = threadIdx.x; i < 3 * A.nbox; i += blockDim.x) s_vb[i] = A.vbox[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const unsigned M = (unsigned)A.M;
  const int64_t npk = *A.npacks;
  unsigned long long c_leaf = 0, c_twig = 0, c_mac = 0;
  for (;;) {
    unsigned b = 0;
    if (lane == 0) b = atomicAdd(A.queue, 1u);
    b = __shfl_sync(0xffffffffu, b, 0);
    if constexpr (kOnly) {
      if ((int)b >= A.over[0]) break;
      b = (unsigned)A.over[1 + b];
    }
    if ((int64_t)b >= npk) break;
    int tl0, len;
    const int64_t t0 = A.pstart[b];
    const bool valid = pack_lane(A.pstart, A.tflag, b, lane, tl0, len);
    if (!__any_sync(0xffffffffu, valid)) {
      if (lane == 0) atomicOr(A.status, ST_INCOMPLETE);  // a pack must start with a tile
      continue;
    }
    const int64_t t = t0 + lane;
    const unsigned tmask = valid ? (((len >= 32) ? 0xffffffffu : ((1u << len) - 1u)) << tl0) : 0u;
    double px = 0, py = 0, pz = 0, e0 = 0, e1 = 0, e2 = 0, ph = 0, w = 0;
    KelbgArgs kel{0.0, A.kinv, A.sqrtpi};
    if (valid) {
      px = A.tx[t]; py = A.ty[t]; pz = A.tz[t];
      if (kLaw == 5) kel.tq = A.tq[t];
      e0 = A.ex[t]; e1 = A.ey[t]; e2 = A.ez[t]; ph = A.pot[t]; w = A.work[t];
    }
    bool complete = true;
    for (int ib = 0; ib < A.nbox; ++ib) {
      const double vx = s_vb[3 * ib], vy = s_vb[3 * ib + 1], vz = s_vb[3 * ib + 2];
      unsigned u = 0, uf = 0;  // tree_walk_single_aux starts at the root (:286)
      int64_t partner = 0;
      for (;;) {
        const unsigned f = __reduce_min_sync(0xffffffffu, valid ? uf : 0xffffffffu);
        if (f >= M) break;
        // the lanes at node f: whole tiles, all at the same node, so they take
        // the same branch below
        const unsigned am = __ballot_sync(0xffffffffu, valid && uf == f);
        if (valid && uf == f) {
          const double4 a = A.nc4[u];
          const int2 mu = A.meta[u];
          const int2 fw = A.fwd[u];
          const int2 ff = A.fwdf[u];
          // d = (x - vbox) - coc (module_tree_walk_simple.f90:328,345)
          const double dx = (px - vx) - a.x, dy = (py - vy) - a.y, dz = (pz - vz) - a.z;
          const double dist2 = (dx * dx + dy * dy) + dz * dz;
          if (mu.y & kLeafFlag) {
            partner += 1;
            if (!cut_off<kCut>(A, dx, dy, dz)) {  // before the work count (:330)
              w += 1.0;
              ++c_leaf;
              if (dist2 > 0.0) {
                double fx, fy, fz, fp;
                law_leaf64<kLaw>(a.w, dx, dy, dz, dist2, A.eps2, fx, fy, fz, fp, kel);
                e0 += fx; e1 += fy; e2 += fz; ph += fp;
              }
            }
            u = (unsigned)fw.y;
            uf = (unsigned)ff.y;
          } else {
            const bool ok = A.theta2 * dist2 > (A.macb ? A.macb[u] : s_bl2[mu.y & 0xff]);
            const unsigned tf = __ballot_sync(am, !ok) & tmask;
            // MAC evaluations stop at the tile's first failing target (:343-370)
            const int first_fail = tf ? __ffs(tf) - 1 : 32;
            if (lane <= first_fail) ++c_mac;
            if (tf == 0) {
              partner += A.nleaves[u];
              if (!cut_off<kCut>(A, dx, dy, dz)) {  // :377
                double m[9];
#pragma unroll
                for (int k = 0; k < 9; ++k) m[k] = A.mom[kMomStride * (int64_t)u + k];
                double fx, fy, fz, fp;
                law_twig64<kLaw>(a.w, m, dx, dy, dz, dist2, A.eps2, fx, fy, fz, fp);
                e0 += fx; e1 += fy; e2 += fz; ph += fp;
                w += 1.0;
                ++c_twig;
              }
              u = (unsigned)fw.y;
              uf = (unsigned)ff.y;
            } else {
              u = (unsigned)fw.x;
              uf = (unsigned)ff.x;
            }
          }
        }
        __syncwarp();
      }
      if (valid && partner != A.npart) complete = false;
    }
    if (valid) {
      A.ex[t] = e0; A.ey[t] = e1; A.ez[t] = e2; A.pot[t] = ph; A.work[t] = w;
    }
    if (__any_sync(0xffffffffu, !complete) && lane == 0) atomicOr(A.status, ST_INCOMPLETE);
  }
  warp_add_counters(A.counters, c_leaf, c_twig, c_mac);
}

// ---------------------------------------------------------------------------
// The same two walks (law 3, no cutoff, one box) by one block per bucket of 32
// targets or pack of tiles, bit for bit: a target's result is the sum of its
// interactions' terms in the order of the walk, and that order is the node order
// (RPO for the per-target walk, forward preorder for tiles).  So the interactions can be
// found and evaluated in any order, as long as each target's terms are added in
// node order:
//  1. the block finds the bucket's interactions from a shared stack of (node, targets that
//     reach it), eight nodes per warp and round, lane = target; a node's accepting targets
//     give one list entry (order index, leaf flag, target mask), the others open it;
//  2. the list is sorted by the order index;
//  3. batches of 32 entries: the (entry, target) pairs are packed, twigs and leaves
//     apart, so that every lane evaluates an interaction; the terms go to shared memory;
//     then one warp per component adds them per target, entry by entry.
// The walks above give a bucket to one warp, a serial chain of dependent loads and FP64
// latencies (4,099 particles are 129 such warps), and evaluate with 77 % of the lanes
// active (here 96 %).
// Lists hold kListCap entries (shared memory: two blocks per SM).  Where scattered
// targets' union is longer, the per-target walk goes on with half as many targets, down
// to kListMin (a target's result does not depend on its bucket); what is still
// too long, and a pack, is left to the walks above (A.over), and so are the block's next 1, 2, 4,
// .. 16 buckets unsearched while this goes on.  16,000 of 100,000 uniform particles in any
// order, theta 0.4: 18.3 ms by warps, 19.0 with whole buckets left to them, 7.0 so; 1,000 of
// 1M Plummer particles, of which four are often too many: 31.1 / 16.7 / 16.3.
constexpr int kListThreads = 256;
constexpr int kListWarps = kListThreads / 32;
constexpr int kListCap = 8192;
constexpr int kListNodes = 8;   // nodes per warp and round
constexpr int kListPop = kListWarps * kListNodes;
// a pop takes at most kListPop entries and each pushes at most 8 (one level down)
constexpr int kListStack = (kMaxLevel + 2) * 8 * kListPop;
constexpr int kListBatch = 32;  // entries per batch
constexpr int kListMin = 4;     // targets

struct __align__(16) ListShared {
  unsigned long long list[kListCap];            // order index << 33 | leaf << 32 | target mask
  double term[kListBatch][4][32];
  uint16_t pair[2][kListBatch * 32];            // twigs, leaves: entry << 5 | target
  double tgt[3][32];
  double bl2[kMaxLevel + 1];
  uint2 cnt[kListWarps];
  unsigned partner[32];
  uint32_t self[2][kListBatch];                 // by batch parity: targets whose own leaf the entry is
  unsigned bucket;
};

template <bool kTile>
__global__ void __launch_bounds__(kListThreads, 2) k_walk_list64(WalkArgs A) {
  extern __shared__ __align__(16) unsigned char dyn[];
  ListShared& S = *reinterpret_cast<ListShared*>(dyn);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  for (int i = tid; i <= kMaxLevel; i += kListThreads) S.bl2[i] = A.bl2[i];
  uint2* stack = A.lstack + (int64_t)blockIdx.x * kListStack;
  const int64_t nbk = *A.tree_status & ST_TIMEOUT ? 0
                      : kTile ? (int64_t)*A.npacks : (A.nt + A.lper - 1) / A.lper;
  const double vx = A.vbox[0], vy = A.vbox[1], vz = A.vbox[2];
  unsigned long long c_leaf = 0, c_twig = 0, c_mac = 0;
  int64_t b = 0, first = 0;  // bucket, and its targets [first, first + left) to do (per target)
  int left = 0;
  int width = kTile ? 32 : A.lper, fits = 0;  // targets at a time, lists in a row that fitted
  int back = 0, skip = 0;                     // buckets to leave unsearched: after a miss, now
  for (;;) {
    if (left == 0) {
      if (tid == 0) S.bucket = atomicAdd(A.queue, 1u);
      __syncthreads();
      b = S.bucket;
      if (b >= nbk) break;
      first = b * A.lper;
      left = kTile ? 1 : (int)min((int64_t)A.lper, A.nt - first);
      if (skip > 0) {
        --skip;
        if (tid == 0) A.over[1 + atomicAdd(A.over, 1)] = kTile ? (int32_t)b : left << kOverShift | (int32_t)first;
        left = 0;
        __syncthreads();
        continue;
      }
    }
    if (tid < 32) S.partner[tid] = 0u;
    bool valid;
    int64_t t0;
    const int len = min(width, left);
    unsigned tmask = 0u;  // the lanes of this lane's tile
    if (kTile) {
      int tl0, len;
      t0 = A.pstart[b];
      valid = pack_lane(A.pstart, A.tflag, b, lane, tl0, len);
      tmask = valid ? (((len >= 32) ? 0xffffffffu : ((1u << len) - 1u)) << tl0) : 0u;
    } else {
      t0 = first;
      valid = lane < len;
    }
    const unsigned all = __ballot_sync(0xffffffffu, valid);
    if (all == 0u) {
      if (tid == 0) atomicOr(A.status, ST_INCOMPLETE);  // a pack must start with a tile
      left = 0;
      __syncthreads();
      continue;
    }
    const int64_t t = t0 + lane;
    double px = 0, py = 0, pz = 0;
    if (valid) {
      px = A.tx[t]; py = A.ty[t]; pz = A.tz[t];
    }
    // x - vbox (module_tree_walk_pthreads.f90:595, module_tree_walk_simple.f90:328)
    const double sx = px - vx, sy = py - vy, sz = pz - vz;
    if (w == 0) {
      S.tgt[0][lane] = sx; S.tgt[1][lane] = sy; S.tgt[2][lane] = sz;
    }
    // ---- 1. the interactions.  Per tile the walk starts at the root
    // (module_tree_walk_simple.f90:286), per target with its children (:601)
    int top, cnt = 0;
    bool over = false;
    {
      const int4 lk = A.drec[0].link;
      const int nch = min(8, lk.y >> 16);
      if (kTile || (lk.y & kLeafFlag)) {
        if (tid == 0) stack[0] = make_uint2(0u, all);
        top = 1;
      } else {
        if (tid < nch) stack[tid] = make_uint2((unsigned)(lk.x + nch - 1 - tid), all);
        top = nch;
      }
    }
    __syncthreads();
    unsigned partner = 0, mac = 0;
    while (top > 0) {
      const int take = min(top, kListPop);
      top -= take;
      uint2 en[kListNodes];
      double4 pos[kListNodes];
      int4 lk[kListNodes];
#pragma unroll
      for (int j = 0; j < kListNodes; ++j) {
        const int i = w * kListNodes + j;
        en[j] = i < take ? stack[top + i] : make_uint2(0u, 0u);
      }
#pragma unroll
      for (int j = 0; j < kListNodes; ++j) {
        const LevelRecord* r = A.drec + en[j].x;
        pos[j] = ld256(&r->pos);
        lk[j] = r->link;
      }
      // lane j keeps node j's decision
      unsigned my_acc = 0, my_open = 0;
      int my_first = 0, my_nch = 0, my_rpo = 0, my_leaf = 0;
#pragma unroll
      for (int j = 0; j < kListNodes; ++j) {
        const unsigned reach = en[j].y;  // 0: no node
        const bool in = (reach >> lane) & 1u;
        const bool leaf = (lk[j].y & kLeafFlag) != 0;
        unsigned acc = reach;
        if (!leaf && reach) {
          const double dx = sx - pos[j].x, dy = sy - pos[j].y, dz = sz - pos[j].z;
          const double dist2 = (dx * dx + dy * dy) + dz * dz;
          const bool ok = A.theta2 * dist2 > (A.macb ? A.macb[lk[j].w] : S.bl2[lk[j].y & 0xff]);
          const unsigned fail = __ballot_sync(0xffffffffu, in && !ok);
          if (kTile) {
            // a tile opens a twig if any of its targets fails; MAC evaluations
            // stop at the first (module_tree_walk_simple.f90:343-370)
            const unsigned tf = fail & tmask;
            if (in && lane <= (tf ? __ffs(tf) - 1 : 32)) ++mac;
            acc = __ballot_sync(0xffffffffu, in && tf == 0u);
          } else {
            if (in) ++mac;
            acc = reach & ~fail;
          }
        }
        if ((acc >> lane) & 1u) partner += leaf ? 1u : (unsigned)lk[j].z;
        if (lane == j) {
          my_acc = acc;
          my_open = reach & ~acc;
          my_first = lk[j].x;
          my_nch = min(8, lk[j].y >> 16);
          my_rpo = lk[j].w;
          my_leaf = leaf ? 1 : 0;
        }
      }
      const unsigned ab = __ballot_sync(0xffffffffu, my_acc != 0u);
      const int npush = my_open ? my_nch : 0;
      int off = npush;  // inclusive over the first kListNodes lanes
#pragma unroll
      for (int o = 1; o < kListNodes; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, off, o);
        if (lane >= o) off += y;
      }
      const int wtotal = __shfl_sync(0xffffffffu, off, kListNodes - 1);
      off -= npush;
      if (lane == 0) S.cnt[w] = make_uint2((unsigned)__popc(ab), (unsigned)wtotal);
      __syncthreads();  // the counts are in; every warp has read its stack entries
      const uint2 c = lane < kListWarps ? S.cnt[lane] : make_uint2(0u, 0u);
      const int lpre = (int)__reduce_add_sync(0xffffffffu, lane < w ? c.x : 0u);
      const int ltot = (int)__reduce_add_sync(0xffffffffu, c.x);
      off += (int)__reduce_add_sync(0xffffffffu, lane < w ? c.y : 0u);
      const int ptot = (int)__reduce_add_sync(0xffffffffu, c.y);
      if (cnt + ltot > kListCap || top + ptot > kListStack) {
        over = true;
        break;
      }
      if (my_acc) {
        const unsigned idx = (unsigned)(kTile ? A.rpo2fpo[my_rpo] : my_rpo);
        S.list[cnt + lpre + __popc(ab & lt)] =
            ((unsigned long long)(idx << 1 | (unsigned)my_leaf) << 32) | my_acc;
      }
      for (int k = 0; k < npush; ++k) stack[top + off + k] = make_uint2((unsigned)(my_first + k), my_open);
      cnt += ltot;
      top += ptot;
      __syncthreads();
    }
    if (over) {
      fits = 0;
      if (!kTile && len > kListMin) {
        width = max(len >> 1, kListMin);
      } else {
        if (tid == 0) A.over[1 + atomicAdd(A.over, 1)] = kTile ? (int32_t)b : left << kOverShift | (int32_t)first;
        left = 0;
        skip = back = min(16, max(1, 2 * back));
      }
      __syncthreads();
      continue;
    }
    back = 0;
    left -= len;
    first += len;
    if (kTile) left = 0;
    else if (++fits >= 16 && width < A.lper) fits = 0, width = min(2 * width, A.lper);
    c_mac += mac;
    atomicAdd(&S.partner[lane], partner);
    // ---- 2. node order: bitonic sort, padded to a power of two
    int P = 64;
    while (P < cnt) P <<= 1;
    for (int i = cnt + tid; i < P; i += kListThreads) S.list[i] = ~0ull;
    __syncthreads();
    for (int k = 2; k <= P; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int i = tid; i < (P >> 1); i += kListThreads) {
          const int lo = ((i & ~(j - 1)) << 1) | (i & (j - 1)), hi = lo | j;
          const unsigned long long x = S.list[lo], y = S.list[hi];
          if ((x > y) == ((lo & k) == 0)) {
            S.list[lo] = y;
            S.list[hi] = x;
          }
        }
        __syncthreads();
      }
    // ---- 3. terms and ordered sums: warps 0..3 add ex, ey, ez, phi, warp 4 work
    double* const out = w == 0 ? A.ex : w == 1 ? A.ey : w == 2 ? A.ez : w == 3 ? A.pot : A.work;
    double sum = 0.0;
    if (w < 5 && valid) sum = out[t];
    int par = 0;
    for (int e0 = 0; e0 < cnt; e0 += kListBatch, par ^= 1) {
      const int ne = min(kListBatch, cnt - e0);
      // pairs: prefix over the batch's entries, then each warp lists four of them
      const unsigned long long en = lane < ne ? S.list[e0 + lane] : 0ull;
      const bool leaf = (en >> 32) & 1u;
      const int nt = leaf ? 0 : __popc((unsigned)en), nl = leaf ? __popc((unsigned)en) : 0;
      int both = nt | (nl << 16);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, both, o);
        if (lane >= o) both += y;
      }
      const int total = __shfl_sync(0xffffffffu, both, 31);
      const int pt = total & 0xffff, pl = total >> 16;
      both -= nt | (nl << 16);
#pragma unroll
      for (int j = 0; j < kListBatch / kListWarps; ++j) {
        const int e = w * (kListBatch / kListWarps) + j;
        const unsigned m = __shfl_sync(0xffffffffu, (unsigned)en, e);
        const int lf = __shfl_sync(0xffffffffu, leaf ? 1 : 0, e);
        const int p0 = __shfl_sync(0xffffffffu, both, e);
        if ((m >> lane) & 1u)
          S.pair[lf][(lf ? p0 >> 16 : p0 & 0xffff) + __popc(m & lt)] = (uint16_t)(e << 5 | lane);
        if (lane == 0) S.self[par][e] = 0u;
      }
      __syncthreads();  // the pairs are listed, and the last batch's terms are added
      for (int i = tid; i < pt; i += kListThreads) {
        const int pr = S.pair[0][i], e = pr >> 5, q = pr & 31;
        const int idx = (int)(S.list[e0 + e] >> 33);
        const int64_t u = kTile ? A.fpo2rpo[idx] : idx;
        const double4 a = ld256(A.nc4 + u);
        const double* mp = A.mom + kMomStride * u;
        const double4 m0 = ld256(mp), m1 = ld256(mp + 4);
        const double m[9] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w, mp[8]};
        const double dx = S.tgt[0][q] - a.x, dy = S.tgt[1][q] - a.y, dz = S.tgt[2][q] - a.z;
        const double dist2 = (dx * dx + dy * dy) + dz * dz;
        double fx, fy, fz, fp;
        law_twig64<3>(a.w, m, dx, dy, dz, dist2, A.eps2, fx, fy, fz, fp);
        S.term[e][0][q] = fx; S.term[e][1][q] = fy; S.term[e][2][q] = fz; S.term[e][3][q] = fp;
      }
      for (int i = tid; i < pl; i += kListThreads) {
        const int pr = S.pair[1][i], e = pr >> 5, q = pr & 31;
        const int idx = (int)(S.list[e0 + e] >> 33);
        const int64_t u = kTile ? A.fpo2rpo[idx] : idx;
        const double4 a = ld256(A.nc4 + u);
        const double dx = S.tgt[0][q] - a.x, dy = S.tgt[1][q] - a.y, dz = S.tgt[2][q] - a.z;
        const double dist2 = (dx * dx + dy * dy) + dz * dz;
        if (dist2 > 0.0) {
          double fx, fy, fz, fp;
          law_leaf64<3>(a.w, dx, dy, dz, dist2, A.eps2, fx, fy, fz, fp);
          S.term[e][0][q] = fx; S.term[e][1][q] = fy; S.term[e][2][q] = fz; S.term[e][3][q] = fp;
        } else {
          atomicOr(&S.self[par][e], 1u << q);
        }
      }
      if (tid == 0) {
        c_twig += (unsigned)pt;
        c_leaf += (unsigned)pl;
      }
      __syncthreads();
      if (w < 4) {
#pragma unroll 8
        for (int e = 0; e < ne; ++e) {
          const unsigned m = (unsigned)S.list[e0 + e] & ~S.self[par][e];
          if ((m >> lane) & 1u) sum += S.term[e][w][lane];
        }
      } else if (w == 4) {
#pragma unroll 8
        for (int e = 0; e < ne; ++e)
          if (((unsigned)S.list[e0 + e] >> lane) & 1u) sum += 1.0;
      }
    }
    if (w < 5 && valid) out[t] = sum;
    if (w == 0 && __any_sync(0xffffffffu, valid && S.partner[lane] != (unsigned)A.npart) && lane == 0)
      atomicOr(A.status, ST_INCOMPLETE);
    __syncthreads();  // the list and the partner counts may be written again
  }
  warp_add_counters(A.counters, c_leaf, c_twig, c_mac);
}

// Greedy packing of consecutive tiles into warps.  The targets are cut into
// chunks of kPackChunk, each chunk's bounds moved forward to the next tile
// start; one warp per chunk steps through its tiles in order and opens a new
// pack whenever the next tile would not fit the 32 lanes.  Two consecutive
// packs hold at least 33 targets between them, so a chunk of kPackChunk + 31
// targets has at most 127 packs (kPackSlots leaves a margin).  The packs are
// then compacted in chunk order into pstart.
constexpr int64_t kPackChunk = 2048;
constexpr int kPackSlots = 256;

// the first tile start at or after p, or nt: a tile holds at most 32
// targets, so one lies in [p, p + 31]
__device__ __forceinline__ int64_t first_tile_start(int64_t p, int64_t nt,
                                                    const int32_t* __restrict__ tflag, int lane) {
  if (p >= nt) return nt;
  const int64_t q = p + lane;
  const unsigned m = __ballot_sync(0xffffffffu, q >= nt || tflag[q] > 0);
  return m ? min(p + __ffs(m) - 1, nt) : nt;
}

__global__ void k_pack_tiles(int64_t nt, const int32_t* __restrict__ tflag,
                             int32_t* __restrict__ raw, int32_t* __restrict__ pcount,
                             uint32_t* status) {
  const int lane = threadIdx.x & 31;
  const int64_t nchunks = (nt + kPackChunk - 1) / kPackChunk;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t ch = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; ch < nchunks;
       ch += nwarps) {
    int64_t p = first_tile_start(ch * kPackChunk, nt, tflag, lane);
    const int64_t e = first_tile_start((ch + 1) * kPackChunk, nt, tflag, lane);
    int k = 0;
    while (p < e && k < kPackSlots) {
      if (lane == 0) raw[ch * kPackSlots + k] = (int32_t)p;
      ++k;
      // the pack ends at the last tile start (or e) in [p + 1, p + 32]
      const int64_t q = p + 1 + lane;
      const unsigned m = __ballot_sync(0xffffffffu, q <= e && (q == e || tflag[q] > 0));
      p = m ? p + 1 + (31 - __clz(m)) : e;
    }
    if (lane == 0) {
      if (p < e) atomicOr(status, ST_INCOMPLETE);
      pcount[ch] = k;
    }
  }
}

__global__ void k_pack_compact(int64_t nt, int64_t nchunks, const int32_t* __restrict__ raw,
                               const int32_t* __restrict__ pcount, const int32_t* __restrict__ poff,
                               int32_t* __restrict__ pstart) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nchunks * kPackSlots;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ch = i / kPackSlots;
    const int k = (int)(i % kPackSlots);
    if (k < pcount[ch]) pstart[poff[ch] + k] = raw[i];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) pstart[poff[nchunks]] = (int32_t)nt;
}

// per-target tile lengths from the compact (first, count) list
__global__ void k_tile_flags(int64_t ntiles, const int2* __restrict__ tiles,
                             int32_t* __restrict__ tflag) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ntiles;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int2 tl = tiles[i];
    tflag[tl.x] = tl.y;
  }
}

__global__ void k_tiles_from_tree(int32_t M, int T, const int32_t* __restrict__ nleaves,
                                  const int32_t* __restrict__ parent,
                                  const int32_t* __restrict__ first_part, int2* tiles,
                                  unsigned int* ntiles) {
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < M;
       u += (int64_t)gridDim.x * blockDim.x) {
    int lv = nleaves[u];
    int p = parent[u];
    if (lv <= T && (p < 0 || nleaves[p] > T)) {
      unsigned slot = atomicAdd(ntiles, 1u);
      tiles[slot] = make_int2(first_part[u], lv);
    }
  }
}

__global__ void k_same_keys(int64_t n, const int64_t* __restrict__ a, const int64_t* __restrict__ b,
                            unsigned int* differ) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    if (a[i] != b[i]) atomicOr(differ, 1u);
}

__global__ void k_reset_counter(unsigned int* q) { *q = 0; }

// calls f(law, cut) with both as compile-time constants (std::integral_constant)
template <class F>
void launch_law_cut(int law, bool cut, F&& f) {
  using T = std::true_type;
  using Fl = std::false_type;
  auto go = [&](auto L) {
    if (cut) f(L, T{});
    else f(L, Fl{});
  };
  if (law == 2) go(std::integral_constant<int, 2>{});
  else if (law == 4) go(std::integral_constant<int, 4>{});
  else if (law == 5) go(std::integral_constant<int, 5>{});
  else go(std::integral_constant<int, 3>{});
}

// mac (coulomb/module_interaction_specific.f90:256-275) for mac_select != 0,
// as a per-twig threshold t with "accept iff theta2 dist2 > t": the Bmax MAC
// has t = min(bmax^2, 3 boxlength2(level)); any other selection accepts
// nothing (the N^2 code), t = +inf.
__global__ void k_mac_thresholds(int64_t M, int mode, const int2* __restrict__ meta,
                                 const double* __restrict__ mom, const double* __restrict__ bl2,
                                 double* __restrict__ macb) {
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < M;
       u += (int64_t)gridDim.x * blockDim.x) {
    const int2 mu = meta[u];
    if (mu.y & kLeafFlag) continue;
    if (mode == 1) {
      const double bmax = mom[kMomStride * u + kMomBmax];
      macb[u] = fmin(bmax * bmax, 3.0 * bl2[mu.y & 0xff]);
    } else {
      macb[u] = INFINITY;
    }
  }
}

}  // namespace

int launch_walk_mixed(Ctx* c, int64_t nt, const double* tx, const double* ty, const double* tz,
                      double* ex, double* ey, double* ez, double* pot, double* work,
                      const int2* tiles, int64_t ntiles, bool per_target, const int32_t* tflag,
                      const int32_t* pstart, const int32_t* npacks, cudaStream_t s, int slot,
                      int64_t shape_nt, bool keyed);

const double* grown_charges_if_same(Ctx* c, int64_t nt, const int64_t* d_tkeys) {
  if (!d_tkeys || nt != c->n) return nullptr;
  unsigned int* d_diff = reinterpret_cast<unsigned int*>(c->d_small + 7);
  unsigned int h_diff = 1;
  cudaMemsetAsync(d_diff, 0, 4, c->stream);
  COUNT_LAUNCH();
  k_same_keys<<<296, 256, 0, c->stream>>>(nt, d_tkeys, c->key.p, d_diff);
  if (!cuda_ok(c, cudaMemcpyAsync(&h_diff, d_diff, 4, cudaMemcpyDeviceToHost, c->stream), "keys") ||
      !cuda_ok(c, cudaStreamSynchronize(c->stream), "keys"))
    return nullptr;
  return h_diff == 0 ? c->q.p : nullptr;
}

int prepare_mac(Ctx* c, const double** macb) {
  *macb = nullptr;
  if (c->prm.mac_select == 0) return PEPCG_OK;
  const int64_t M = c->nnodes;
  if (!ensure(c, c->macb, M, "mac thresholds")) return PEPCG_ERR_OOM;
  COUNT_LAUNCH();
  const unsigned g = (unsigned)((M + 255) / 256 > 148 * 16 ? 148 * 16 : (M + 255) / 256);
  k_mac_thresholds<<<g, 256, 0, c->stream>>>(M, c->prm.mac_select, c->meta.p, c->mom.p,
                                             c->d_box + 9, c->macb.p);
  if (!cuda_ok(c, cudaGetLastError(), "mac thresholds")) return PEPCG_ERR_CUDA;
  *macb = c->macb.p;
  return PEPCG_OK;
}

// Whether the plain walk of nt targets goes by k_walk_list64: while its buckets of 32
// are fewer than the warps that the walks by warp keep resident (2,960 per target, 96
// registers and five blocks of four warps per SM; 3,552 per tile), and where a list
// is likely to fit (theta >= 0.35, or a tree smaller than a list).  Walk ms, by warp ->
// by lists, per target: 1,000 particles 0.237 -> 0.082, 4,099: 0.46 -> 0.117, 16,411
// (Plummer, theta 0.4) 3.36 -> 1.22, 40,009: 0.86 -> 0.56; per tile 4,099: 0.46 -> 0.133, 40,009:
// 1.10 -> 0.69.  With more buckets the lists' own work (sort, packing, a
// node per warp step in the search: 480 instructions per 32 interactions, 158 of them
// FP64) costs more than idle lanes: 100,003: 3.04 against 3.43, 250,000: 6.4 against 9.0.
// Targets without keys may lie in any order: their line is lower, since scattered targets
// share few nodes (theta 0.4, of 100,000 Plummer particles: 4,000 targets 20.0 -> 4.1, 16,000:
// 24.0 -> 14.0, in proportion from there on, against 24.5 by warps for 64,000; on a line
// through them 64,000 targets 3.9 by warps, 4.4 by lists).
constexpr int64_t kListTargets = 65536;
constexpr int64_t kListOthers = 24576;
constexpr int kListBlocks = 148 * 2;
static bool use_list_walk(const Ctx* c, int64_t nt, bool keyed, bool chunked, bool packed) {
  const pepcg_params& p = c->prm;
  if (p.precision != PEPCG_PRECISION_PLAIN || chunked || p.force_law != 3 || has_spatial_cutoff(p) ||
      c->nboxes != 1)
    return false;
  if (p.walk != PEPCG_WALK_PER_TARGET && !packed) return false;
  if (nt > (keyed ? kListTargets : kListOthers)) return false;
  return c->nnodes <= kListCap || (p.mac_select == 0 && p.theta2 >= 0.12);
}

// Targets per bucket of the per-target walk: a bucket's search and its batches are a
// serial chain, so few targets take small buckets, as long as two blocks per SM hold
// them all.  Walk ms with 32 / 16 / 8: 1,000 targets 0.078 / 0.065 / 0.057, 4,099: 0.116 /
// 0.090 / 0.120, 8,000: 0.133 / 0.166 / 0.227.
static int list_bucket(int64_t nt) {
  return nt <= 8 * kListBlocks ? 8 : nt <= 16 * kListBlocks ? 16 : 32;
}

// What the host needs of a finished walk, into mapped host memory (two or three
// device-to-host copies to pageable memory and their staging took 10 us more).
static __global__ void k_walk_summary(const unsigned long long* __restrict__ ctr,
                                      const uint32_t* __restrict__ status,
                                      const uint32_t* __restrict__ tree_status,
                                      const int32_t* __restrict__ over, Ctx::GrowSummary* out) {
  if (threadIdx.x < 3) out->ctr[threadIdx.x] = ctr[threadIdx.x];
  if (threadIdx.x == 3) out->walk_status = *status | *tree_status;
  if (threadIdx.x == 4) out->nover = over ? *over : 0;
}

int traverse_device(Ctx* c, int64_t nt, const double* tx, const double* ty, const double* tz,
                    const int64_t* tkeys, bool self, double* ex, double* ey, double* ez,
                    double* pot, double* work, const double* tq, const ChunkPlan* plan,
                    int64_t shape_nt, bool keyed) {
  if (!c->has_tree) {
    c->err = "traverse called without a grown tree";
    return PEPCG_ERR_NO_TREE;
  }
  if (nt <= 0) return PEPCG_OK;
  if (c->prm.force_law == 5 && !tq) {
    c->err = "force_law 5 (Kelbg) needs the targets' charges: traverse the grown particles "
             "(pepcg_traverse_self_device, pepcg_traverse_range_device, or pepcg_traverse_tree "
             "with the grown keys)";
    return PEPCG_ERR_UNSUPPORTED;
  }
  keyed = keyed || self || tkeys;
  cudaStream_t s = c->stream;
  const int walk = c->prm.walk;
  // bucket queues, counters, barrier words and the status word
  if (!cuda_ok(c, cudaMemsetAsync(c->d_small + 8, 0, 13 * sizeof(unsigned long long), s), "walk state"))
    return PEPCG_ERR_CUDA;
  int64_t ntiles = 0;
  if (walk == PEPCG_WALK_PER_TILE) {
    const int T = c->prm.tile_size < 1 ? 1 : (c->prm.tile_size > 32 ? 32 : c->prm.tile_size);
    bool from_tree = self;
    if (!self && tkeys && nt == c->n) {
      unsigned int* d_diff = reinterpret_cast<unsigned int*>(c->d_small + 4);
      unsigned int h_diff = 1;
      cudaMemsetAsync(d_diff, 0, 4, s);
      COUNT_LAUNCH();
      k_same_keys<<<296, 256, 0, s>>>(nt, tkeys, c->key.p, d_diff);
      if (!cuda_ok(c, cudaMemcpyAsync(&h_diff, d_diff, 4, cudaMemcpyDeviceToHost, s), "tiles") ||
          !cuda_ok(c, cudaStreamSynchronize(s), "tiles"))
        return PEPCG_ERR_CUDA;
      from_tree = (h_diff == 0);
    }
    if (!ensure(c, c->tiles, 2 * (nt + 1), "tiles")) return PEPCG_ERR_OOM;
    int2* d_tiles = reinterpret_cast<int2*>(c->tiles.p);
    if (from_tree) {
      unsigned int* d_nt = reinterpret_cast<unsigned int*>(c->d_small + 5);
      unsigned int h_nt = 0;
      cudaMemsetAsync(d_nt, 0, 4, s);
      COUNT_LAUNCH();
      k_tiles_from_tree<<<296, 256, 0, s>>>((int32_t)c->nnodes, T, c->nleaves_ptr(), c->parent.p,
                                            c->first_part.p, d_tiles, d_nt);
      if (!cuda_ok(c, cudaMemcpyAsync(&h_nt, d_nt, 4, cudaMemcpyDeviceToHost, s), "tiles") ||
          !cuda_ok(c, cudaStreamSynchronize(s), "tiles"))
        return PEPCG_ERR_CUDA;
      ntiles = h_nt;
    } else {
      int rc = host_tiles(c, nt, tkeys, T, d_tiles, &ntiles);
      if (rc) return rc;
    }
  }
  // per-tile walk: several whole tiles per warp.  Measured at 4M (Plummer,
  // theta 0.4): the packed FP64 walk beats one tile per warp at every tile
  // size (32: 278 vs 851 ms); in the mixed form the wide group kernel with
  // tiles as buckets wins at 32 targets (127 vs 148 ms) and loses at 24
  // (167 vs 146 ms)
  const bool packed = walk == PEPCG_WALK_PER_TILE &&
                      (c->prm.precision == PEPCG_PRECISION_PLAIN || c->prm.tile_size <= 24);
  const int32_t* pstart = nullptr;
  const int32_t* npacks = nullptr;
  if (packed) {
    if (!ensure(c, c->tflag, nt, "tile flags")) return PEPCG_ERR_OOM;
    if (!cuda_ok(c, cudaMemsetAsync(c->tflag.p, 0, nt * sizeof(int32_t), s), "tile flags"))
      return PEPCG_ERR_CUDA;
    COUNT_LAUNCH();
    k_tile_flags<<<296, 256, 0, s>>>(ntiles, reinterpret_cast<const int2*>(c->tiles.p),
                                     c->tflag.p);
    // packs of whole tiles, <= 32 targets each
    const int64_t nch = (nt + kPackChunk - 1) / kPackChunk;
    const int64_t ntmp = (nch + 1 + 2047) / 2048 + 1;
    const int64_t cap = nch * kPackSlots + 1;  // packs + the end; every slot may be used
    if (!ensure(c, c->tpack, (size_t)(nch * kPackSlots + 2 * (nch + 1) + ntmp + cap), "packs"))
      return PEPCG_ERR_OOM;
    int32_t* raw = c->tpack.p;
    int32_t* pcount = raw + nch * kPackSlots;
    int32_t* poff = pcount + nch + 1;
    int32_t* tmp = poff + nch + 1;
    int32_t* ps = tmp + ntmp;
    pstart = ps;
    npacks = poff + nch;
    if (!cuda_ok(c, cudaMemsetAsync(pcount, 0, (nch + 1) * sizeof(int32_t), s), "packs"))
      return PEPCG_ERR_CUDA;
    const unsigned gw = (unsigned)std::min<int64_t>((nch * 32 + 255) / 256, 148 * 8);
    COUNT_LAUNCH();
    k_pack_tiles<<<gw, 256, 0, s>>>(nt, c->tflag.p, raw, pcount, c->d_status);
    exclusive_scan_i32(pcount, poff, nch + 1, tmp, s);
    const unsigned gc = (unsigned)std::min<int64_t>((nch * kPackSlots + 255) / 256, 148 * 8);
    COUNT_LAUNCH();
    k_pack_compact<<<gc, 256, 0, s>>>(nt, nch, raw, pcount, poff, ps);
  }
  const int nchunks = plan ? plan->nchunks : 1;
  if (nchunks > 1) {
    bool ok = walk != PEPCG_WALK_PER_TILE && !c->far_field && nchunks <= Ctx::kMaxChunks &&
              plan->bounds[0] == 0 && plan->bounds[nchunks] == nt;
    for (int k = 1; ok && k < nchunks; ++k)
      ok = plan->bounds[k] % c->group_size() == 0 && plan->bounds[k] >= plan->bounds[k - 1];
    if (!ok) {
      c->err = "traverse: invalid chunk plan";
      return PEPCG_ERR_BAD_ARG;
    }
  }
  WalkArgs A;
  A.nc4 = c->nc4.p;
  A.meta = c->meta.p;
  A.fwd = c->fwd.p;
  A.mom = c->mom.p;
  A.nleaves = c->nleaves_ptr();
  A.bl2 = c->d_box + 9;
  {
    int rc = prepare_mac(c, &A.macb);
    if (rc) return rc;
  }
  A.vbox = c->d_vbox;
  A.nbox = c->nboxes;
  A.theta2 = c->prm.theta2;
  A.eps2 = c->prm.eps2;
  A.M = (int32_t)c->nnodes;
  A.npart = c->n;
  A.counters = c->counters;
  A.status = c->d_status;
  A.queue = c->walk_queue();
  A.tiles = reinterpret_cast<const int2*>(c->tiles.p);
  A.ntiles = ntiles;
  A.kinv = c->prm.kelbg_invsqrttemp;
  A.sqrtpi = std::sqrt(std::acos(-1.0));
  A.fwdf = c->fwdf.p;
  A.tflag = c->tflag.p;
  A.pstart = pstart;
  A.npacks = npacks;
  A.has_cut = has_spatial_cutoff(c->prm) ? 1 : 0;
  for (int k = 0; k < 3; ++k) A.cut[k] = c->prm.spatial_interaction_cutoff[k];
  const int blocks = 148 * 8;
  const bool lists = use_list_walk(c, nt, keyed, plan != nullptr, packed);
  if (lists) {
    A.lper = list_bucket(nt);
    const int64_t nbk = packed ? (nt + kPackChunk - 1) / kPackChunk * kPackSlots
                               : (nt + A.lper - 1) / A.lper;
    if (!ensure(c, c->wstack, (size_t)2 * kListStack * kListBlocks, "walk stacks") ||
        !ensure(c, c->over, 1 + (packed ? nbk : (int64_t)nt), "walk lists"))
      return PEPCG_ERR_OOM;
    A.drec = c->drec.p;
    A.tree_status = c->d_tree_status;
    A.rpo2fpo = c->rpo2fpo.p;
    A.fpo2rpo = c->fpo2rpo.p;
    A.lstack = reinterpret_cast<uint2*>(c->wstack.p);
    A.over = c->over.p;
    if (!cuda_ok(c, cudaMemsetAsync(c->over.p, 0, sizeof(int32_t), s), "walk lists"))
      return PEPCG_ERR_CUDA;
  }
  // chunks alternate between the context stream and walk2, so that each
  // chunk's walk starts while the previous one finishes its last buckets
  const bool two = nchunks > 1;  // a plan comes with walk2 (copy_streams)
  if (two && (!cuda_ok(c, cudaEventRecord(c->fork, s), "fork") ||
              !cuda_ok(c, cudaStreamWaitEvent(c->walk2, c->fork, 0), "fork")))
    return PEPCG_ERR_CUDA;
  for (int k = 0; k < nchunks; ++k) {
    const int64_t t0 = nchunks > 1 ? plan->bounds[k] : 0;
    const int64_t t1 = nchunks > 1 ? plan->bounds[k + 1] : nt;
    const int slot = two ? (k & 1) : 0;
    const cudaStream_t sk = slot ? c->walk2 : s;
    A.queue = c->walk_queue(slot);
    if (plan && plan->ready && !cuda_ok(c, cudaStreamWaitEvent(sk, plan->ready[k], 0), "chunk wait"))
      return PEPCG_ERR_CUDA;
    if (k == 0) cudaEventRecord(c->ev[5], s);
    if (t1 > t0) {
      A.nt = t1 - t0;
      A.tx = tx + t0; A.ty = ty + t0; A.tz = tz + t0;
      A.ex = ex + t0; A.ey = ey + t0; A.ez = ez + t0; A.pot = pot + t0; A.work = work + t0;
      A.tq = tq ? tq + t0 : nullptr;
      if (k >= 2) {  // a chunk's queue again (the first two are zero)
        COUNT_LAUNCH();
        k_reset_counter<<<1, 1, 0, sk>>>(A.queue);
      }
      if (c->prm.precision == PEPCG_PRECISION_PLAIN) {
        COUNT_LAUNCH();
        const int law = c->prm.force_law;
        const bool cut = A.has_cut != 0;
        if (lists) {
          auto kern = packed ? k_walk_list64<true> : k_walk_list64<false>;
          if (!cuda_ok(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)sizeof(ListShared)), "list walk"))
            return PEPCG_ERR_CUDA;
          kern<<<kListBlocks, kListThreads, sizeof(ListShared), sk>>>(A);
        } else if (walk == PEPCG_WALK_PER_TARGET) {
          launch_law_cut(law, cut, [&](auto L, auto C) {
            k_walk_target64<decltype(L)::value, decltype(C)::value><<<blocks, kWalkThreads, 0, sk>>>(A);
          });
        } else if (packed) {
          launch_law_cut(law, cut, [&](auto L, auto C) {
            k_walk_tilepack64<decltype(L)::value, decltype(C)::value><<<blocks, kWalkThreads, 0, sk>>>(A);
          });
        } else {
          if (walk == PEPCG_WALK_GROUP) A.tiles = nullptr;
          if (walk == PEPCG_WALK_GROUP && c->group_size() == 64) {
            launch_law_cut(law, cut, [&](auto L, auto C) {
              k_walk_tile64<decltype(L)::value, 2, decltype(C)::value><<<blocks, kWalkThreads, 0, sk>>>(A);
            });
          } else {
            launch_law_cut(law, cut, [&](auto L, auto C) {
              k_walk_tile64<decltype(L)::value, 1, decltype(C)::value><<<blocks, kWalkThreads, 0, sk>>>(A);
            });
          }
        }
      } else {
        int rc = launch_walk_mixed(c, t1 - t0, A.tx, A.ty, A.tz, A.ex, A.ey, A.ez, A.pot, A.work,
                                   walk == PEPCG_WALK_PER_TILE ? A.tiles : nullptr, ntiles,
                                   walk == PEPCG_WALK_PER_TARGET, packed ? c->tflag.p : nullptr,
                                   pstart, npacks, sk, slot, shape_nt > 0 ? shape_nt : nt, keyed);
        if (rc) return rc;
      }
      if (!cuda_ok(c, cudaGetLastError(), "walk launch")) return PEPCG_ERR_CUDA;
    }
    if (plan && plan->done) cudaEventRecord(plan->done[k], sk);
  }
  if (two && (!cuda_ok(c, cudaEventRecord(c->join, c->walk2), "join") ||
              !cuda_ok(c, cudaStreamWaitEvent(s, c->join, 0), "join")))
    return PEPCG_ERR_CUDA;
  cudaEventRecord(c->ev[6], s);
  if (c->far_field) {
    int rc = lattice_add(c, nt, tx, ty, tz, ex, ey, ez, pot, false);
    if (rc) return rc;
  }
  cudaEventRecord(c->ev[7], s);
  if (plan && plan->before_sync && !plan->before_sync()) return PEPCG_ERR_CUDA;
  auto summary = [&]() {
    COUNT_LAUNCH();
    k_walk_summary<<<1, 32, 0, s>>>(c->counters, c->d_status, c->d_tree_status, lists ? c->over.p : nullptr, c->d_sum);
    return cuda_ok(c, cudaGetLastError(), "walk summary") &&
           cuda_ok(c, cudaStreamSynchronize(s), "walk");
  };
  if (!summary()) return PEPCG_ERR_CUDA;
  if (lists && c->h_sum->nover > 0) {  // lists that did not fit: these buckets by the warp walks
    COUNT_LAUNCH();
    k_reset_counter<<<1, 1, 0, s>>>(A.queue);
    COUNT_LAUNCH();
    if (packed) k_walk_tilepack64<3, false, true><<<blocks, kWalkThreads, 0, s>>>(A);
    else k_walk_target64<3, false, true><<<blocks, kWalkThreads, 0, s>>>(A);
    cudaEventRecord(c->ev[6], s);
    cudaEventRecord(c->ev[7], s);
    if (!summary()) return PEPCG_ERR_CUDA;
  }
  const unsigned long long* ctr = c->h_sum->ctr;
  const uint32_t st = c->h_sum->walk_status;
  c->st.leaf_interactions = (int64_t)ctr[0];
  c->st.twig_interactions = (int64_t)ctr[1];
  c->st.interactions = (int64_t)(ctr[0] + ctr[1]);
  c->st.mac_evaluations = (int64_t)ctr[2];
  float ms = 0;
  if (cudaEventElapsedTime(&ms, c->ev[5], c->ev[6]) == cudaSuccess) c->st.t_walk_ms = ms;
  if (cudaEventElapsedTime(&ms, c->ev[6], c->ev[7]) == cudaSuccess) c->st.t_lattice_ms = ms;
  if (st) return status_to_code(c, st);
  return take_adjoint_status(c);
}

}  // namespace pepcg
