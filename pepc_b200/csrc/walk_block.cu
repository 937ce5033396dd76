// walk_block.cu -- the 64-target group walk and its adjoint with one thread
// block (or a cluster of blocks) per target bucket, for walks of few buckets
// (block_walk_shape has the lines).
//
// k_walk_group64 and k_adj_group64 (walk_mixed.cu) give each bucket to one warp,
// whose traversal is a serial chain of dependent loads and batches: with fewer
// buckets than resident warps (2,960) most of the chip idles and the call takes
// the longest bucket's chain, and with up to three times as many buckets in key order
// the last of them still do.  Here the W warps of a block share one bucket:
//  - one traversal stack per block (global memory): a round pops up to 32 W
//    nodes, one per thread, decided exactly as there (the same FP32
//    group-centred opening test), so the lists are the same;
//  - accepted twigs and leaves go to rings in shared memory at positions from a
//    prefix over the block's warps (fixed order: results do not vary from run to
//    run), and when a ring holds 32 W records every warp evaluates 32 of them at
//    the same time, the remainder being divided evenly at the end;
//  - each warp sums its records for all 64 targets (FP32 within a batch of at most
//    32, then FP64), and the warps' FP64 sums are added in warp order.
// With still fewer buckets a cluster of S blocks shares one: every block runs
// the same first rounds until the stack holds kSplitAt S nodes, keeps every S-th
// of them, and the blocks' sums meet through distributed shared memory.
// Periodic walks push the roots of all image boxes at once (the box index in
// the stack entry's upper bits), so that 27 boxes cost no 27 chains of rounds.
#include <cooperative_groups.h>

#include <algorithm>

#include "mixed.cuh"

namespace cg = cooperative_groups;

namespace pepcg {

namespace {

constexpr int kSplitAt = 24;      // stacked nodes per cluster block before they are divided
constexpr int kBoxShift = 25;     // stack entry: node | box << 25 (trees below 2^25 nodes)

// what the traversal reads, of either kernel's arguments
struct BlockTree {
  const LevelRecord* drec;
  const double* macb;
  float theta2;
  double theta2d;
};

// the bucket's targets as a lane sees them
struct BucketLane {
  Targets64 T;  // sxa.. without a box vector
  bool v0, v1;
  unsigned vm0, vm1;
  double gx, gy, gz;  // group centre
  float rg;           // radius of the sphere around it that holds every target
  float hx, hy, hz;   // half edges of the box around it that holds every target
  int cnt;            // targets of the bucket
};

__device__ __forceinline__ BucketLane load_bucket(const double* __restrict__ tx,
                                                  const double* __restrict__ ty,
                                                  const double* __restrict__ tz, int64_t t0,
                                                  int cnt, int lane) {
  BucketLane b;
  b.v0 = lane < cnt;
  b.v1 = lane + 32 < cnt;
  b.vm0 = __ballot_sync(0xffffffffu, b.v0);
  b.vm1 = __ballot_sync(0xffffffffu, b.v1);
  const int64_t ta = t0 + lane, tb = t0 + 32 + lane;
  double pa[3] = {0, 0, 0}, pb[3] = {0, 0, 0}, lo[3], hi[3];
  if (b.v0) { pa[0] = tx[ta]; pa[1] = ty[ta]; pa[2] = tz[ta]; }
  if (b.v1) { pb[0] = tx[tb]; pb[1] = ty[tb]; pb[2] = tz[tb]; }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = b.v0 ? pa[d] : INFINITY;
    hi[d] = b.v0 ? pa[d] : -INFINITY;
    if (b.v1) {
      lo[d] = fmin(lo[d], pb[d]);
      hi[d] = fmax(hi[d], pb[d]);
    }
    for (int o = 16; o > 0; o >>= 1) {
      lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
      hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
    }
  }
  b.gx = 0.5 * (lo[0] + hi[0]);
  b.gy = 0.5 * (lo[1] + hi[1]);
  b.gz = 0.5 * (lo[2] + hi[2]);
  Targets64& T = b.T;
  T.rxa = (float)(pa[0] - b.gx); T.rya = (float)(pa[1] - b.gy); T.rza = (float)(pa[2] - b.gz);
  T.rxb = (float)(pb[0] - b.gx); T.ryb = (float)(pb[1] - b.gy); T.rzb = (float)(pb[2] - b.gz);
  T.sxa = pa[0]; T.sya = pa[1]; T.sza = pa[2];
  T.sxb = pb[0]; T.syb = pb[1]; T.szb = pb[2];
  float rg = fmaxf(b.v0 ? sqrtf(T.rxa * T.rxa + T.rya * T.rya + T.rza * T.rza) : 0.f,
                   b.v1 ? sqrtf(T.rxb * T.rxb + T.ryb * T.ryb + T.rzb * T.rzb) : 0.f);
  for (int o = 16; o > 0; o >>= 1) rg = fmaxf(rg, __shfl_xor_sync(0xffffffffu, rg, o));
  // the sphere and the box must contain every target after rounding
  b.rg = rg * 1.0001f + 1e-30f;
  b.hx = (float)(0.5 * (hi[0] - lo[0])) * 1.0001f + 1e-30f;
  b.hy = (float)(0.5 * (hi[1] - lo[1])) * 1.0001f + 1e-30f;
  b.hz = (float)(0.5 * (hi[2] - lo[2])) * 1.0001f + 1e-30f;
  b.cnt = cnt;
  return b;
}

// A decided node as its thread hands it to the staging callbacks
struct Decided {
  float cx, cy, cz;  // centre minus the group centre (the box vector included)
  double4 a;         // centre and charge
  int4 lk;           // links of its level record
  int node;          // level-order position
  int box;
};

// One sweep: the boxes [ib0, ib0 + nb) of the bucket's walk, by the whole block
// (part of nparts blocks).  leaf(slot, d) and twig(slot, d) stage a record;
// flush_twigs(head, n) / flush_leaves(head, n) evaluate n <= 32 W records
// between two block barriers.  Every thread of the block takes the same rounds.
// The stack is bounded as in k_walk_group_wide: a pop takes at most 32 W entries
// and each pushes at most 8.
template <int W, bool kStrict, class Leaf, class Twig, class FT, class FL>
__device__ __forceinline__ bool block_traverse(const BlockTree& B, const BucketLane& K,
                                               const float* s_bl2, const double* s_bl2d,
                                               const double* s_vb, uint2* s_cnt, int* stack,
                                               int ib0, int nb, int part, int nparts,
                                               unsigned long long& c_mac, int64_t& partner,
                                               Leaf&& leaf, Twig&& twig, FT&& flush_twigs,
                                               FL&& flush_leaves) {
  constexpr int kThreads = 32 * W;
  constexpr int kCap = W * kStackCap;
  constexpr int kMask = 2 * kThreads - 1;  // rings of 64 W records
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const float theta2 = B.theta2;
  int nT = 0, hT = 0, nL = 0, hL = 0;
  int top = nb;
  bool mine = part == 0;  // before the stack is divided only the first block records
  bool divided = nparts == 1;
  if (nparts == 1) mine = true;
  for (int i = tid; i < nb; i += kThreads) stack[i] = (int)((unsigned)i << kBoxShift);
  __syncthreads();
  while (top > 0) {
    const int take = top < kThreads ? top : kThreads;
    top -= take;
    const unsigned ent = tid < take ? (unsigned)stack[top + tid] : 0u;
    bool isleaf = false, accept = false, open = false, amb = false;
    float bl = 0.f;
    double bld = 0.0;
    Decided d;
    d.cx = d.cy = d.cz = 0.f;
    d.a = make_double4(0, 0, 0, 0);
    d.lk = make_int4(0, 0, 0, 0);
    d.node = nb > 1 ? (int)(ent & ((1u << kBoxShift) - 1u)) : (int)ent;
    d.box = nb > 1 ? (int)(ent >> kBoxShift) : 0;
    if (tid < take) {
      const LevelRecord* rec = B.drec + d.node;
      d.a = ld256(&rec->pos);
      d.lk = rec->link;
      const double* v = s_vb + 3 * (ib0 + d.box);
      d.cx = (float)(d.a.x - (K.gx - v[0]));
      d.cy = (float)(d.a.y - (K.gy - v[1]));
      d.cz = (float)(d.a.z - (K.gz - v[2]));
      if (d.lk.y & kLeafFlag) {
        isleaf = true;
      } else {
        bl = B.macb ? (float)B.macb[d.lk.w] : s_bl2[d.lk.y & 0xff];
        const float dc = sqrtf(d.cx * d.cx + d.cy * d.cy + d.cz * d.cz);
        float dmin = dc - K.rg, dmax = dc + K.rg;
        if constexpr (kStrict) {
          // conservative: the sphere decides only where the FP64 test of
          // every target certainly agrees
          bld = B.macb ? B.macb[d.lk.w] : s_bl2d[d.lk.y & 0xff];
          dmin = dc * (1.0f - 1e-5f) - K.rg;
          dmax = dc * (1.0f + 1e-5f) + K.rg;
        }
        if (dmin > 0.f && theta2 * (dmin * dmin) > bl) accept = true;
        else if (!(theta2 * (dmax * dmax) > bl)) open = true;
        else amb = true;
        if (mine && !amb) c_mac += 1;
        if (amb) {
          // no target is nearer than the box: accepted without a test per target
          // (counted as one test each, as the tests below would)
          const float ax = fmaxf(fabsf(d.cx) - K.hx, 0.f), ay = fmaxf(fabsf(d.cy) - K.hy, 0.f),
                      az = fmaxf(fabsf(d.cz) - K.hz, 0.f);
          if (theta2 * ((ax * ax + ay * ay + az * az) * (1.0f - 1e-5f)) > bl) {
            amb = false;
            accept = true;
            if (mine) c_mac += (unsigned)K.cnt;
          }
        }
      }
    }
    unsigned am = __ballot_sync(0xffffffffu, amb);
    while (am) {
      const int j = __ffs(am) - 1;
      am &= am - 1;
      bool fa, fb;
      if constexpr (kStrict) {
        // mac (coulomb/module_interaction_specific.f90:256-275) in FP64, in
        // the reference's operation order: theta2 * dist2 > boxlength2; a
        // strict sweep covers one box, whose vector T already holds
        const double ux = __shfl_sync(0xffffffffu, d.a.x, j);
        const double uy = __shfl_sync(0xffffffffu, d.a.y, j);
        const double uz = __shfl_sync(0xffffffffu, d.a.z, j);
        const double ub = __shfl_sync(0xffffffffu, bld, j);
        double dx = K.T.sxa - ux, dy = K.T.sya - uy, dz = K.T.sza - uz;
        double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
        fa = K.v0 && !(__dmul_rn(B.theta2d, d2) > ub);
        dx = K.T.sxb - ux; dy = K.T.syb - uy; dz = K.T.szb - uz;
        d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
        fb = K.v1 && !(__dmul_rn(B.theta2d, d2) > ub);
      } else {
        const float ux = __shfl_sync(0xffffffffu, d.cx, j);
        const float uy = __shfl_sync(0xffffffffu, d.cy, j);
        const float uz = __shfl_sync(0xffffffffu, d.cz, j);
        const float ub = __shfl_sync(0xffffffffu, bl, j);
        const float2 dx = __fadd2_rn(make_float2(K.T.rxa, K.T.rxb), f2(-ux)),
                     dy = __fadd2_rn(make_float2(K.T.rya, K.T.ryb), f2(-uy)),
                     dz = __fadd2_rn(make_float2(K.T.rza, K.T.rzb), f2(-uz));
        const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
        fa = K.v0 && !(theta2 * d2.x > ub);
        fb = K.v1 && !(theta2 * d2.y > ub);
      }
      const unsigned f0 = __ballot_sync(0xffffffffu, fa);
      const unsigned f1 = __ballot_sync(0xffffffffu, fb);
      if (lane == j) {
        accept = (f0 | f1) == 0;
        open = !accept;
        // MAC evaluations up to the first failing target, in target order
        if (mine)
          c_mac += (unsigned)(f0 ? __popc(K.vm0 & ((2u << (__ffs(f0) - 1)) - 1u))
                                 : __popc(K.vm0) + (f1 ? __popc(K.vm1 & ((2u << (__ffs(f1) - 1)) - 1u))
                                                       : __popc(K.vm1)));
      }
    }
    const unsigned lb = __ballot_sync(0xffffffffu, isleaf && mine);
    const unsigned ab = __ballot_sync(0xffffffffu, accept && mine);
    const int npush = open ? min(8, d.lk.y >> 16) : 0;
    int wtotal;
    int off = warp_excl_scan8(npush, lt, wtotal);
    if (lane == 0) s_cnt[w] = make_uint2((unsigned)__popc(lb) | ((unsigned)__popc(ab) << 16), (unsigned)wtotal);
    __syncthreads();  // the counts are in; every thread has read its stack entry
    const uint2 c = lane < W ? s_cnt[lane] : make_uint2(0u, 0u);
    const unsigned pre = __reduce_add_sync(0xffffffffu, lane < w ? c.x : 0u);
    const unsigned tot = __reduce_add_sync(0xffffffffu, c.x);
    off += (int)__reduce_add_sync(0xffffffffu, lane < w ? c.y : 0u);
    const int total = (int)__reduce_add_sync(0xffffffffu, c.y);
    if (top + total > kCap) return false;  // cannot happen within the bound; every thread leaves
    if (isleaf && mine) {
      leaf((hL + nL + (int)(pre & 0xffffu) + __popc(lb & lt)) & kMask, d);
      partner += 1;
    }
    if (accept && mine) {
      twig((hT + nT + (int)(pre >> 16) + __popc(ab & lt)) & kMask, d);
      partner += d.lk.z;
    }
    nL += (int)(tot & 0xffffu);
    nT += (int)(tot >> 16);
    if (npush > 0) {
      int* dst = stack + top + off;
      const unsigned box = nb > 1 ? (unsigned)d.box << kBoxShift : 0u;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < npush) dst[k] = (int)((unsigned)(d.lk.x + k) | box);
    }
    top += total;
    const bool ft = nT >= kThreads, fl = nL >= kThreads;
    if (ft) cp_async_wait_all();
    __syncthreads();  // stack entries and staged records are visible to the block
    if (ft) {
      flush_twigs(hT, kThreads);
      hT = (hT + kThreads) & kMask;
      nT -= kThreads;
    }
    if (fl) {
      flush_leaves(hL, kThreads);
      hL = (hL + kThreads) & kMask;
      nL -= kThreads;
    }
    if (!divided && top >= kSplitAt * nparts) {
      // every block has the same stack: keep the entries part, part + nparts, ...
      const int keep = (top - part + nparts - 1) / nparts;
      for (int i0 = 0; i0 < keep; i0 += kThreads) {
        const int i = i0 + tid;
        const int e = i < keep ? stack[i * nparts + part] : 0;
        __syncthreads();
        if (i < keep) stack[i] = e;
        __syncthreads();
      }
      top = keep;
      divided = mine = true;
    }
  }
  cp_async_wait_all();
  __syncthreads();
  if (nT > 0) flush_twigs(hT, nT);
  if (nL > 0) flush_leaves(hL, nL);
  __syncthreads();  // the rings and the stack may be written again
  return true;
}

template <int W, bool kStrict>
constexpr size_t walk_block_smem() {
  return 64 * W * (sizeof(TwigRec64<kStrict>) + sizeof(StagedLeaf)) + 8 * 32 * W * sizeof(double) +
         4 * 64 * sizeof(double);
}

// Resident blocks per SM: 1 of sixteen warps, 2 of eight; five of four warps where 96
// registers do (the default form: 200,003 particles 1.69 -> 1.60 ms against four blocks).
template <int W, bool kStrict>
constexpr int walk_block_resident() {
  return W == 16 ? 1 : W == 8 ? 2 : kStrict ? 4 : 5;
}

template <int W, bool kStrict>
__global__ void __launch_bounds__(32 * W, walk_block_resident<W, kStrict>())
    k_walk_block64(MixArgs A, int* __restrict__ gstack, int nparts, int sweep) {
  constexpr int kThreads = 32 * W;
  constexpr int kRingB = 2 * kThreads;
  __shared__ float s_bl2[kMaxLevel + 1];
  __shared__ double s_bl2d[kMaxLevel + 1];
  __shared__ double s_vb[3 * 125];
  __shared__ uint2 s_cnt[W];
  __shared__ int64_t s_part[W];
  __shared__ int64_t s_sum[2];  // partners and records of this block
  __shared__ unsigned s_bucket;
  extern __shared__ __align__(16) unsigned char dyn[];
  TwigRec64<kStrict>* rt = reinterpret_cast<TwigRec64<kStrict>*>(dyn);
  StagedLeaf* rl = reinterpret_cast<StagedLeaf*>(rt + kRingB);
  double* s_acc = reinterpret_cast<double*>(rl + kRingB);  // [8][kThreads]
  double* s_out = s_acc + 8 * kThreads;                    // [4][64]: the block's sums
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (int i = tid; i <= kMaxLevel; i += kThreads) {
    s_bl2[i] = (float)A.bl2[i];
    s_bl2d[i] = A.bl2[i];
  }
  for (int i = tid; i < 3 * A.nbox; i += kThreads) s_vb[i] = A.vbox[i];
  int* stack = gstack + (int64_t)blockIdx.x * W * kStackCap;
  const int part = nparts > 1 ? (int)(blockIdx.x % nparts) : 0;
  const int64_t nbuckets = *A.tree_status & ST_TIMEOUT ? 0 : (A.nt + 63) / 64;
  const BlockTree B{A.drec, A.macb, A.theta2, A.theta2d};
  unsigned long long c_leaf = 0, c_twig = 0, c_mac = 0;
  for (bool first = true;; first = false) {
    // a bucket from the queue, or (clusters: one bucket each) the cluster's
    if (nparts > 1) {
      if (!first) break;
      if (tid == 0) s_bucket = blockIdx.x / nparts;
    } else if (tid == 0) {
      s_bucket = atomicAdd(A.queue, 1u);
    }
    __syncthreads();
    const int64_t b = s_bucket;
    if (b >= nbuckets) break;
    const int64_t t0 = b * 64;
    const int cnt = (int)min((int64_t)64, A.nt - t0);
    const int64_t ta = t0 + lane, tb = t0 + 32 + lane;
    BucketLane K = load_bucket(A.tx, A.ty, A.tz, t0, cnt, lane);
    double* acc = s_acc + tid;
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k * kThreads] = 0.0;
    int64_t partner = 0, records = 0;
    bool complete = true;
    const double pa[3] = {K.T.sxa, K.T.sya, K.T.sza}, pb[3] = {K.T.sxb, K.T.syb, K.T.szb};
    for (int ib0 = 0; ib0 < A.nbox && complete; ib0 += sweep) {
      const int nb = min(sweep, A.nbox - ib0);
      if constexpr (kStrict) {  // shifted positions x - vbox (one box per sweep)
        const double* v = s_vb + 3 * ib0;
        K.T.sxa = pa[0] - v[0]; K.T.sya = pa[1] - v[1]; K.T.sza = pa[2] - v[2];
        K.T.sxb = pb[0] - v[0]; K.T.syb = pb[1] - v[1]; K.T.szb = pb[2] - v[2];
      }
      complete = block_traverse<W, kStrict>(
          B, K, s_bl2, s_bl2d, s_vb, s_cnt, stack, ib0, nb, part, nparts, c_mac, partner,
          [&](int slot, const Decided& d) {
            StagedLeaf& r = rl[slot];
            r.c = make_float4(d.cx, d.cy, d.cz, (float)d.a.w);
            r.x = d.a.x; r.y = d.a.y; r.z = d.a.z;
            r.box = ib0 + d.box;
          },
          [&](int slot, const Decided& d) {
            TwigRec64<kStrict>& r = rt[slot];
            if constexpr (kStrict) {
              r.cx = d.a.x;
              r.cy = d.a.y;
              r.cz = d.a.z;
            } else {
              r.c = make_float4(-d.cx, -d.cy, -d.cz, (float)d.a.w);
            }
            const float4* m = A.mom32 + kMom32Stride * (int64_t)d.lk.w;
            cp_async16(&r.m0, m);
            cp_async16(&r.m1, m + 1);
            cp_async16(&r.m2, m + 2);
          },
          [&](int head, int n) {
            records += n;
            const int share = (n + W - 1) / W, s0 = w * share, m = min(share, n - s0);
            if (m <= 0 || !K.v0) return;
            twig_batch64<kStrict>(rt, (head + s0) & (kRingB - 1), m, kRingB, K.T, A.eps2, acc, kThreads);
            c_twig += (unsigned)m * (K.v1 ? 2u : 1u);
          },
          [&](int head, int n) {
            records += n;
            const int share = (n + W - 1) / W, s0 = w * share, m = min(share, n - s0);
            if (m <= 0 || !K.v0) return;
            const unsigned self = leaf_batch64<kStrict>(
                rl, (head + s0) & (kRingB - 1), m, kRingB, K.T, K.v1, A, ta, tb,
                [&](const StagedLeaf& r) {
                  const double* v = s_vb + 3 * r.box;
                  return make_double3(v[0], v[1], v[2]);
                },
                acc, kThreads);
            c_leaf += (unsigned)m * (K.v1 ? 2u : 1u) - self;
          });
    }
    for (int o = 16; o > 0; o >>= 1) partner += __shfl_xor_sync(0xffffffffu, partner, o);
    if (lane == 0) s_part[w] = complete ? partner : -1;
    __syncthreads();
    // the block's sums, warps in order
    for (int i = tid; i < 256; i += kThreads) {
      const int k = i >> 6, t = i & 63;
      const double* a = s_acc + (4 * (t >> 5) + k) * kThreads + (t & 31);
      double s = a[0];
#pragma unroll
      for (int v = 1; v < W; ++v) s += a[32 * v];
      s_out[i] = s;
    }
    if (tid == 0) {
      int64_t p = 0;
      for (int v = 0; v < W; ++v) p = (p < 0 || s_part[v] < 0) ? -1 : p + s_part[v];
      s_sum[0] = p;
      s_sum[1] = records;
    }
    if (nparts > 1) cg::this_cluster().sync();
    else __syncthreads();
    if (part == 0) {
      int64_t p = 0, rec = 0;
      for (int s = 0; s < nparts; ++s) {
        const int64_t* o = nparts > 1 ? cg::this_cluster().map_shared_rank(s_sum, s) : s_sum;
        p = (p < 0 || o[0] < 0) ? -1 : p + o[0];
        rec += o[1];
      }
      for (int i = tid; i < 4 * cnt; i += kThreads) {
        const int k = i / cnt, t = i - k * cnt;
        double* out = k == 0 ? A.ex : k == 1 ? A.ey : k == 2 ? A.ez : A.pot;
        double v = out[t0 + t];
        for (int s = 0; s < nparts; ++s) {
          const double* o = nparts > 1 ? cg::this_cluster().map_shared_rank(s_out, s) : s_out;
          v += o[64 * k + t];
        }
        out[t0 + t] = v;
      }
      for (int t = tid; t < cnt; t += kThreads) A.work[t0 + t] += (double)rec;
      if (tid == 0 && p != A.npart * A.nbox) atomicOr(A.status, ST_INCOMPLETE);
    }
    if (nparts > 1) cg::this_cluster().sync();  // the sums stay in place until they are read
    else __syncthreads();
  }
  warp_add3(A.counters, c_leaf, c_twig, c_mac);
}

template <int W, bool kWithE>
constexpr size_t adj_block_smem() {
  return 64 * W * (sizeof(StagedTwig) + sizeof(StagedLeafA)) + 32 * (kWithE ? 4 : 2) * sizeof(float4);
}

// The adjoint on the same lists: records staged as in k_adj_group64, evaluated
// transposed (lane = record) against the bucket's targets in shared memory.
template <int W, bool kWithE>
__global__ void __launch_bounds__(32 * W, W == 16 ? 1 : (W == 8 ? 2 : 4))
    k_adj_block64(AdjMixArgs A, int* __restrict__ gstack, int nparts, int sweep) {
  constexpr int kThreads = 32 * W;
  constexpr int kRingB = 2 * kThreads;
  __shared__ float s_bl2[kMaxLevel + 1];
  __shared__ double s_vb[3 * 125];
  __shared__ uint2 s_cnt[W];
  __shared__ int64_t s_part[W];
  __shared__ int64_t s_sum;
  __shared__ unsigned s_bucket;
  extern __shared__ __align__(16) unsigned char dyn[];
  StagedTwig* rt = reinterpret_cast<StagedTwig*>(dyn);
  StagedLeafA* rl = reinterpret_cast<StagedLeafA*>(rt + kRingB);
  float4(*tg)[kWithE ? 4 : 2] = reinterpret_cast<float4(*)[kWithE ? 4 : 2]>(rl + kRingB);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (int i = tid; i <= kMaxLevel; i += kThreads) s_bl2[i] = (float)A.bl2[i];
  for (int i = tid; i < 3 * A.nbox; i += kThreads) s_vb[i] = A.vbox[i];
  int* stack = gstack + (int64_t)blockIdx.x * W * kStackCap;
  const int part = nparts > 1 ? (int)(blockIdx.x % nparts) : 0;
  const int64_t nbuckets = (A.nt + 63) / 64;
  const BlockTree B{A.drec, A.macb, A.theta2, 0.0};
  const float2 E2 = f2(A.eps2);
  unsigned long long c_leaf = 0, c_twig = 0, c_mac = 0;
  for (bool first = true;; first = false) {
    if (nparts > 1) {
      if (!first) break;
      if (tid == 0) s_bucket = blockIdx.x / nparts;
    } else if (tid == 0) {
      s_bucket = atomicAdd(A.queue, 1u);
    }
    __syncthreads();
    const int64_t b = s_bucket;
    if (b >= nbuckets) break;
    const int64_t t0 = b * 64;
    const int cnt = (int)min((int64_t)64, A.nt - t0);
    const BucketLane K = load_bucket(A.tx, A.ty, A.tz, t0, cnt, lane);
    const unsigned nvalid = (unsigned)cnt;
    if (w == 0) {
      const int64_t ta = t0 + lane, tb = t0 + 32 + lane;
      const float gpa = K.v0 ? (float)A.gphi[ta] : 0.f, gpb = K.v1 ? (float)A.gphi[tb] : 0.f;
      // an absent target sits far away with zero gradients: it adds exact zeros
      tg[lane][0] = make_float4(K.v0 ? K.T.rxa : 1e10f, K.v1 ? K.T.rxb : 1e10f,
                                K.v0 ? K.T.rya : 1e10f, K.v1 ? K.T.ryb : 1e10f);
      tg[lane][1] = make_float4(K.v0 ? K.T.rza : 1e10f, K.v1 ? K.T.rzb : 1e10f, gpa, gpb);
      if constexpr (kWithE) {
        tg[lane][2] = make_float4(K.v0 ? (float)A.gex[ta] : 0.f, K.v1 ? (float)A.gex[tb] : 0.f,
                                  K.v0 ? (float)A.gey[ta] : 0.f, K.v1 ? (float)A.gey[tb] : 0.f);
        tg[lane][3] = make_float4(K.v0 ? (float)A.gez[ta] : 0.f, K.v1 ? (float)A.gez[tb] : 0.f, 0.f, 0.f);
      }
    }
    int64_t partner = 0;
    bool complete = true;
    for (int ib0 = 0; ib0 < A.nbox && complete; ib0 += sweep) {
      const int nb = min(sweep, A.nbox - ib0);
      complete = block_traverse<W, false>(
          B, K, s_bl2, nullptr, s_vb, s_cnt, stack, ib0, nb, part, nparts, c_mac, partner,
          [&](int slot, const Decided& d) {
            StagedLeafA& r = rl[slot];
            r.c = make_float4(d.cx, d.cy, d.cz, (float)d.a.w);
            r.x = d.a.x; r.y = d.a.y; r.z = d.a.z;
            r.node = d.node;
            r.pad = ib0 + d.box;
          },
          [&](int slot, const Decided& d) {
            StagedTwig& r = rt[slot];
            r.c = make_float4(-d.cx, -d.cy, -d.cz, __int_as_float(d.node));
            const float4* m = A.mom32 + kMom32Stride * (int64_t)d.lk.w;
            cp_async16(&r.m0, m);
            cp_async16(&r.m1, m + 1);
            cp_async16(&r.m2, m + 2);
          },
          [&](int head, int n) {
            if (tid < n) {
              adj_twig_record<kWithE>(rt[(head + tid) & (kRingB - 1)], tg, E2, A.adj);
              c_twig += nvalid;
            }
          },
          [&](int head, int n) {
            if (tid < n) {
              const StagedLeafA& r = rl[(head + tid) & (kRingB - 1)];
              const double* v = s_vb + 3 * r.pad;
              adj_leaf_record<kWithE>(r, tg, E2, A, t0, make_double3(v[0], v[1], v[2]));
              c_leaf += nvalid;
            }
          });
    }
    for (int o = 16; o > 0; o >>= 1) partner += __shfl_xor_sync(0xffffffffu, partner, o);
    if (lane == 0) s_part[w] = complete ? partner : -1;
    __syncthreads();
    if (tid == 0) {
      int64_t p = 0;
      for (int v = 0; v < W; ++v) p = (p < 0 || s_part[v] < 0) ? -1 : p + s_part[v];
      s_sum = p;
    }
    if (nparts > 1) cg::this_cluster().sync();
    else __syncthreads();
    if (part == 0 && tid == 0) {
      int64_t p = 0;
      for (int s = 0; s < nparts; ++s) {
        const int64_t o = nparts > 1 ? *cg::this_cluster().map_shared_rank(&s_sum, s) : s_sum;
        p = (p < 0 || o < 0) ? -1 : p + o;
      }
      if (p != A.npart * A.nbox) atomicOr(A.status, ST_INCOMPLETE);
    }
    if (nparts > 1) cg::this_cluster().sync();
    else __syncthreads();
  }
  warp_add3(A.counters, c_leaf, c_twig, c_mac);
}

// grid of `blocks` blocks in clusters of nparts; false: refused (the launchers below pass
// it on, and the walk goes by one warp per bucket)
template <class K, class A>
bool launch_block(Ctx* c, K kern, int threads, size_t smem, int blocks, int nparts, cudaStream_t s,
                  const A& args, int* stack, int sweep) {
  if ((c->refuse & kRefuseCluster) && nparts > 1) return false;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)nparts;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = nparts > 1 ? 1 : 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaLaunchKernelEx(&cfg, kern, args, stack, nparts, sweep) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  COUNT_LAUNCH();
  return true;
}

}  // namespace

// Measured (walk ms, Plummer, theta 0.4, one warp per bucket -> the choice here):
// 16 buckets 0.182 -> 0.042, 64: 0.48 -> 0.064, 141: 0.74 -> 0.114, 257: 1.10 -> 0.20,
// 516: 1.31 -> 0.33, 938: 1.42 -> 0.52, 1,563: 1.54 -> 0.86, 3,126: 1.77 -> 1.60, 6,250:
// 3.42 -> 3.24, and past that one warp per bucket is faster (12,500: 6.46 against 6.56;
// strict: 3,126: 2.48 -> 2.24, 6,250 level).  Eight warps at two blocks per SM beat sixteen
// except for 75 .. 148 buckets, which leave an SM one block each (141 buckets: 0.114
// against 0.137 in clusters of two); four warps from 600 buckets on (516: 0.37 against
// 0.33, 938: 0.52 against 0.58).  The adjoint: 4,688 buckets 6.2 against 6.7 ms.
// Few buckets on a large tree are scattered targets with long lists: sixteen warps
// and eight blocks (8 buckets, 262,144 sources: 0.135 against 0.18 ms).
// Walked targets without keys (keyed false) may lie in any order, and buckets of
// scattered targets are alike: the walk by warps then loses nothing to a longest bucket,
// only to its last wave.  Random and evenly spread targets, targets on a line, of or among
// 100,000 and 1M particles, theta 0.4 and 0.6, time by warps / by blocks:
//   default form  4,063 buckets 0.90 .. 1.05, 4,400: 0.95 .. 1.07, 5,469: 0.94 .. 1.12, 8,594:
//                 0.92 .. 1.02; up to 4,096 none of the cells is slower than the walk by
//                 warps was before both were tuned, from 4,400 some are (0.93 .. 0.97);
//   strict form   2,200 buckets 1.01 .. 1.20, 2,300: 0.92 .. 1.14, 2,368, which fill one wave of
//                 its resident warps: 0.92 .. 1.13, 2,375: 0.99 .. 1.29, 2,960: 1.00 .. 1.19.
bool block_walk_shape(int64_t nt, int64_t npart, BlockWalk kind, bool keyed, BlockShape* sh) {
  const int64_t nb = (nt + 63) / 64;
  if (nb > (kind == BlockWalk::kStrict ? 5000 : kind == BlockWalk::kAdjoint ? 6000 : keyed ? 9000 : 4096))
    return false;
  if (kind == BlockWalk::kStrict && !keyed && nb > 2200 && nb <= 148 * 4 * kWW) return false;
  if (nb <= 18 && npart >= 32768) *sh = {16, 8};
  else if (nb <= 37) *sh = {8, 8};
  else if (nb <= 74) *sh = {8, 4};
  else if (nb <= 148) *sh = {16, 1};
  else if (nb <= 600) *sh = {8, 1};
  else *sh = {4, 1};
  return true;
}

// One cluster per bucket, or resident blocks that take buckets from the queue.
static int block_grid(const BlockShape& sh, int64_t nt, int per_sm) {
  const int64_t nb = (nt + 63) / 64;
  if (sh.parts > 1) return (int)(nb * sh.parts);
  return (int)std::min<int64_t>(nb, 148 * per_sm);
}

bool launch_walk_block64(Ctx* c, const MixArgs& A, const BlockShape& sh, bool strict, int* stack,
                         cudaStream_t s) {
  const int sweep = (!strict && A.M <= (1 << kBoxShift)) ? A.nbox : 1;
  auto go = [&](auto kern, int W, size_t smem) {
    const int per_sm = W == 16 ? 1 : W == 8 ? 2 : strict ? 4 : 5;
    return launch_block(c, kern, 32 * W, smem, block_grid(sh, A.nt, per_sm), sh.parts, s, A, stack, sweep);
  };
  if (sh.warps == 16)
    return strict ? go(k_walk_block64<16, true>, 16, walk_block_smem<16, true>())
                  : go(k_walk_block64<16, false>, 16, walk_block_smem<16, false>());
  if (sh.warps == 8)
    return strict ? go(k_walk_block64<8, true>, 8, walk_block_smem<8, true>())
                  : go(k_walk_block64<8, false>, 8, walk_block_smem<8, false>());
  return strict ? go(k_walk_block64<4, true>, 4, walk_block_smem<4, true>())
                : go(k_walk_block64<4, false>, 4, walk_block_smem<4, false>());
}

bool launch_adj_block64(Ctx* c, const AdjMixArgs& A, const BlockShape& sh, bool with_e, int* stack,
                        cudaStream_t s) {
  const int sweep = c->nnodes <= (1 << kBoxShift) ? A.nbox : 1;
  auto go = [&](auto kern, int W, size_t smem) {
    const int per_sm = W == 16 ? 1 : W == 8 ? 2 : 4;
    return launch_block(c, kern, 32 * W, smem, block_grid(sh, A.nt, per_sm), sh.parts, s, A, stack, sweep);
  };
  if (sh.warps == 16)
    return with_e ? go(k_adj_block64<16, true>, 16, adj_block_smem<16, true>())
                  : go(k_adj_block64<16, false>, 16, adj_block_smem<16, false>());
  if (sh.warps == 8)
    return with_e ? go(k_adj_block64<8, true>, 8, adj_block_smem<8, true>())
                  : go(k_adj_block64<8, false>, 8, adj_block_smem<8, false>());
  return with_e ? go(k_adj_block64<4, true>, 4, adj_block_smem<4, true>())
                : go(k_adj_block64<4, false>, 4, adj_block_smem<4, false>());
}

}  // namespace pepcg
