// walk_mixed.cu -- the mixed-precision walks.
//
// Precision contract.  Every interaction offset is formed in FP64 from the
// FP64 positions and then rounded to FP32; the interaction (monopole + dipole
// + quadrupole, Plummer softened) is evaluated in FP32 with rsqrt; per target
// the FP32 sums of each batch of <= 32 interactions are added to FP64
// accumulators; node moments are computed in FP64 by the upward pass and
// rounded to FP32 once per grow (k_upward_level in grow.cu).
//  * Group walk: the offsets of the target and of the node centre from the
//    group centre g (the centre of the 32 targets' bounding box) are each
//    formed in FP64 and rounded once; the interaction offset is their FP32
//    difference.  Against the FP64 offset rounded once, the extra error is at
//    most 2u (|t - g| + |d|) with u = 2^-24: 2u (1 + r_g/|d|) relative, r_g
//    the group radius.  A leaf whose FP32 offset is exactly zero is re-tested
//    in FP64, so the self test is the reference's dist2 == 0.
//  * Per-target walk: target minus node centre in FP64, then rounded.
//
// The FP32 twig interaction is the reference's quadrupole kernel
// (coulomb/module_coulomb_kernels.f90:60-145) rewritten in the equivalent
// form
//   phi = q/r - (d.p)/r^3 + 3 (d.M.d)/r^5 - tr(Q)/r^3
//   E   = d [q/r^3 - 3 (d.p)/r^5 + 15 (d.M.d)/r^7 - 3 tr(Q)/r^5] + p/r^3 - 6 (M.d)/r^5
// with M = [[qxx, qxy/2, qzx/2], [qxy/2, qyy, qyz/2], [qzx/2, qyz/2, qzz]]
// (expanding the reference's fdx.. / pre2x.. terms gives exactly these
// polynomials), which needs 39 FP32 operations instead of ~130.

#include "mixed.cuh"

namespace pepcg {

namespace {

// Group walk (GROUP and PER_TILE modes): per-tile semantics
// (module_tree_walk_simple.f90:256-384) -- a twig is accepted only if every
// target of the warp's group passes the Barnes-Hut MAC, else it is opened --
// with a wide traversal.  The traversal pops up to 32 nodes from a per-warp
// LIFO stack (global memory) and lane k decides node k:
//   leaf -> queued for evaluation;
//   twig -> the group's bounding sphere decides most nodes at once (every
//           target farther than the MAC distance: accept; none: open); the
//           rest get the exact test one node at a time across the warp
//           (lane = target, a ballot of the failures); opened twigs push
//           their children (child8 table).
// A popped node's centre, level, leaf count and child table are loaded in
// one round.  The MAC is evaluated on the FP32 group-centred offsets, and
// the same offsets go straight into the node's staging record: accepted
// twigs and leaves are written into per-warp ring buffers in shared memory
// at decision time (the twig moments by cp.async), so a batch of 32 is
// evaluated without a load on its critical path; every lane then reads all
// staged records by broadcast.
// Stack bound: a pop takes <= 32 entries and pushes <= 8 per node, so the
// stack never holds more than (kMaxLevel + 1) * 8 * 32 entries; kStackCap
// leaves a margin and an overflow sets ST_INCOMPLETE instead of writing past it.
__global__ void __launch_bounds__(kMixThreads, 5)
    k_walk_group_wide(MixArgs A, int* __restrict__ gstack, const int4* __restrict__ child8,
                      const int* __restrict__ nchild) {
  __shared__ float s_bl2[kMaxLevel + 1];
  __shared__ double s_vb[3 * 125];
  __shared__ StagedTwig s_tw[kWW][kRing];
  __shared__ StagedLeaf s_lf[kWW][kRing];
  for (int i = threadIdx.x; i <= kMaxLevel; i += blockDim.x) s_bl2[i] = (float)A.bl2[i];
  for (int i = threadIdx.x; i < 3 * A.nbox; i += blockDim.x) s_vb[i] = A.vbox[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  int* stack = gstack + (int64_t)(blockIdx.x * kWW + w) * kStackCap;
  StagedTwig* stw = s_tw[w];
  StagedLeaf* stl = s_lf[w];
  const float theta2 = A.theta2;
  const int64_t nbuckets = A.tiles ? A.ntiles : (A.nt + 31) / 32;
  unsigned long long c_leaf = 0, c_twig = 0, c_mac = 0;
  for (;;) {
    unsigned b = 0;
    if (lane == 0) b = atomicAdd(A.queue, 1u);
    b = __shfl_sync(0xffffffffu, b, 0);
    if ((int64_t)b >= nbuckets) break;
    int64_t t0;
    int cnt;
    if (A.tiles) {
      const int2 tl = A.tiles[b];
      t0 = tl.x;
      cnt = tl.y;
    } else {
      t0 = (int64_t)b * 32;
      cnt = (int)min((int64_t)32, A.nt - t0);
    }
    const bool valid = lane < cnt;
    const unsigned vmask = __ballot_sync(0xffffffffu, valid);
    const int64_t t = t0 + lane;
    double px = 0, py = 0, pz = 0;
    double E0 = 0, E1 = 0, E2 = 0, PH = 0, W = 0;
    if (valid) {
      px = A.tx[t]; py = A.ty[t]; pz = A.tz[t];
      E0 = A.ex[t]; E1 = A.ey[t]; E2 = A.ez[t]; PH = A.pot[t]; W = A.work[t];
    }
    // group centre (FP64) and the targets' offsets from it (FP32)
    double lo[3] = {valid ? px : INFINITY, valid ? py : INFINITY, valid ? pz : INFINITY};
    double hi[3] = {valid ? px : -INFINITY, valid ? py : -INFINITY, valid ? pz : -INFINITY};
#pragma unroll
    for (int d = 0; d < 3; ++d)
      for (int o = 16; o > 0; o >>= 1) {
        lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
        hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
      }
    const double g0x = 0.5 * (lo[0] + hi[0]), g0y = 0.5 * (lo[1] + hi[1]), g0z = 0.5 * (lo[2] + hi[2]);
    const float rx = (float)(px - g0x), ry = (float)(py - g0y), rz = (float)(pz - g0z);
    float rg = valid ? sqrtf(rx * rx + ry * ry + rz * rz) : 0.f;
    for (int o = 16; o > 0; o >>= 1) rg = fmaxf(rg, __shfl_xor_sync(0xffffffffu, rg, o));
    rg = rg * 1.0001f + 1e-30f;  // the sphere must contain every target after rounding
    bool complete = true;
    for (int ib = 0; ib < A.nbox; ++ib) {
      const double vx = s_vb[3 * ib], vy = s_vb[3 * ib + 1], vz = s_vb[3 * ib + 2];
      const double sx = px - vx, sy = py - vy, sz = pz - vz;
      const double gx = g0x - vx, gy = g0y - vy, gz = g0z - vz;
      int64_t partner = 0;  // leaves covered by this lane's nodes (summed over the warp at the end)
      int nT = 0, hT = 0, nL = 0, hL = 0;  // ring counts and heads
      int top = 1;
      if (lane == 0) stack[0] = 0;  // the root (walk_simple starts at the root, :286)
      __syncwarp();
      // evaluates the n staged twigs / leaves at the ring heads
      auto flush_twigs = [&](int n) {
        cp_async_wait_all();
        __syncwarp();
        if (valid) {
          float ax = 0.f, ay = 0.f, az = 0.f, ap = 0.f;
          // the batch is at most two contiguous runs of the ring
          const int n1 = min(n, kRing - hT);
          const StagedTwig* r = stw + hT;
#pragma unroll 16
          for (int j = 0; j < n1; ++j) {
            const float4 c = r[j].c;
            twig32(r[j].m0, r[j].m1, r[j].m2, rx - c.x, ry - c.y, rz - c.z, A.eps2, ax, ay, az, ap);
          }
#pragma unroll 8
          for (int j = 0; j < n - n1; ++j) {
            const float4 c = stw[j].c;
            twig32(stw[j].m0, stw[j].m1, stw[j].m2, rx - c.x, ry - c.y, rz - c.z, A.eps2, ax, ay,
                   az, ap);
          }
          E0 += (double)ax; E1 += (double)ay; E2 += (double)az; PH += (double)ap;
          c_twig += (unsigned)n;
        }
        W += (double)n;
        hT = (hT + n) & (kRing - 1);
        nT -= n;
        __syncwarp();
      };
      auto flush_leaves = [&](int n) {
        __syncwarp();
        if (valid) {
          float ax = 0.f, ay = 0.f, az = 0.f, ap = 0.f;
          auto leaf = [&](const StagedLeaf& r) {
            const float4 c = r.c;
            float dx = rx - c.x, dy = ry - c.y, dz = rz - c.z;
            if (dx == 0.f && dy == 0.f && dz == 0.f) {
              // self (dist2 == 0 in FP64) or two points closer than the FP32
              // resolution at the group scale: decide and evaluate in FP64
              const double ex = sx - r.x, ey = sy - r.y, ez = sz - r.z;
              if (ex == 0.0 && ey == 0.0 && ez == 0.0) return;
              dx = (float)ex; dy = (float)ey; dz = (float)ez;
            }
            leaf32(c.w, dx, dy, dz, A.eps2, ax, ay, az, ap);
            ++c_leaf;
          };
          // the batch is at most two contiguous runs of the ring
          const int n1 = min(n, kRing - hL);
          const StagedLeaf* r = stl + hL;
#pragma unroll 8
          for (int j = 0; j < n1; ++j) leaf(r[j]);
#pragma unroll 4
          for (int j = 0; j < n - n1; ++j) leaf(stl[j]);
          E0 += (double)ax; E1 += (double)ay; E2 += (double)az; PH += (double)ap;
        }
        W += (double)n;
        hL = (hL + n) & (kRing - 1);
        nL -= n;
        __syncwarp();
      };
      while (top > 0) {
        const int take = top < 32 ? top : 32;
        top -= take;
        const int node = lane < take ? stack[top + lane] : -1;
        __syncwarp();
        bool isleaf = false, accept = false, open = false, amb = false;
        float cx = 0.f, cy = 0.f, cz = 0.f, bl = 0.f;
        double4 a = make_double4(0, 0, 0, 0);
        int nlv = 0, nch = 0;
        int4 c0 = make_int4(0, 0, 0, 0), c1 = c0;
        if (node >= 0) {
          // one round of loads: what accept, open and leaf each need
          a = A.nc4[node];
          const int2 mu = A.meta[node];
          nlv = A.nleaves[node];
          nch = nchild[node];
          c0 = child8[2 * (int64_t)node];
          c1 = child8[2 * (int64_t)node + 1];
          cx = (float)(a.x - gx); cy = (float)(a.y - gy); cz = (float)(a.z - gz);
          if (mu.y & kLeafFlag) {
            isleaf = true;
          } else {
            bl = A.macb ? (float)A.macb[node] : s_bl2[mu.y & 0xff];
            const float dc = sqrtf(cx * cx + cy * cy + cz * cz);
            const float dmin = dc - rg, dmax = dc + rg;
            if (dmin > 0.f && theta2 * (dmin * dmin) > bl) {
              accept = true;  // every target is farther than dmin
              c_mac += 1;
            } else if (!(theta2 * (dmax * dmax) > bl)) {
              open = true;    // no target can pass
              c_mac += 1;
            } else {
              amb = true;
            }
          }
        }
        // the exact MAC for the undecided nodes, one node at a time across
        // the targets (lane = target): accepted iff no target fails
        unsigned am = __ballot_sync(0xffffffffu, amb);
        while (am) {
          const int j = __ffs(am) - 1;
          am &= am - 1;
          const float ux = __shfl_sync(0xffffffffu, cx, j);
          const float uy = __shfl_sync(0xffffffffu, cy, j);
          const float uz = __shfl_sync(0xffffffffu, cz, j);
          const float ub = __shfl_sync(0xffffffffu, bl, j);
          const float dx = rx - ux, dy = ry - uy, dz = rz - uz;
          const bool fail = valid && !(theta2 * fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > ub);
          const unsigned f = __ballot_sync(0xffffffffu, fail);
          if (lane == j) {
            accept = (f == 0);
            open = !accept;
            // MAC evaluations up to the first failing target, in target order
            c_mac += (unsigned)__popc(f ? (vmask & ((2u << (__ffs(f) - 1)) - 1u)) : vmask);
          }
        }
        const unsigned lb = __ballot_sync(0xffffffffu, isleaf);
        const unsigned ab = __ballot_sync(0xffffffffu, accept);
        if (isleaf) {
          StagedLeaf& r = stl[(hL + nL + __popc(lb & lt)) & (kRing - 1)];
          r.c = make_float4(cx, cy, cz, (float)a.w);
          r.x = a.x; r.y = a.y; r.z = a.z;
          partner += 1;
        }
        if (accept) {
          StagedTwig& r = stw[(hT + nT + __popc(ab & lt)) & (kRing - 1)];
          r.c = make_float4(cx, cy, cz, (float)a.w);
          const float4* m = A.mom32 + kMom32Stride * (int64_t)node;
          cp_async16(&r.m0, m);
          cp_async16(&r.m1, m + 1);
          cp_async16(&r.m2, m + 2);
          partner += nlv;
        }
        nL += __popc(lb);
        nT += __popc(ab);
        // push the children of opened twigs
        const int npush = open ? min(8, nch) : 0;
        int total;
        const int off = warp_excl_scan(npush, lane, total);
        if (top + total > kStackCap) {
          complete = false;  // cannot happen within the bound above
          break;
        }
        if (npush > 0) {
          int* dst = stack + top + off;
          dst[0] = c0.x;
          if (npush > 1) dst[1] = c0.y;
          if (npush > 2) dst[2] = c0.z;
          if (npush > 3) dst[3] = c0.w;
          if (npush > 4) dst[4] = c1.x;
          if (npush > 5) dst[5] = c1.y;
          if (npush > 6) dst[6] = c1.z;
          if (npush > 7) dst[7] = c1.w;
        }
        top += total;
        __syncwarp();
        if (nT >= 32) flush_twigs(32);
        if (nL >= 32) flush_leaves(32);
      }
      if (nT > 0) flush_twigs(nT);
      if (nL > 0) flush_leaves(nL);
      for (int o = 16; o > 0; o >>= 1) partner += __shfl_xor_sync(0xffffffffu, partner, o);
      if (partner != A.npart) complete = false;
    }
    if (valid) {
      A.ex[t] = E0; A.ey[t] = E1; A.ez[t] = E2; A.pot[t] = PH; A.work[t] = W;
    }
    if (__any_sync(0xffffffffu, !complete) && lane == 0) atomicOr(A.status, ST_INCOMPLETE);
  }
  cp_async_wait_all();
  warp_add3(A.counters, c_leaf, c_twig, c_mac);
}

// Group walk over buckets of 64 key-consecutive targets (group_size 64), two
// per lane: lane k holds targets t0 + k and t0 + 32 + k.  The traversal, the
// MAC rule (a twig is accepted only if all 64 targets pass) and the staging
// are those of k_walk_group_wide.  Each staged record is read from shared
// memory once for both of the lane's targets, and the twig interactions of
// the pair run as packed FP32 (twig32x2).  Twig records store the node's
// offset from the group centre negated, so that the pair's offsets are one
// packed add.  Against 32-target buckets the larger group is opened more
// often (about 9 % more interactions at 4M, theta 0.4); the packed pair
// arithmetic and the halved traversal per target more than pay for it.
//
// A round's latency chain and instructions matter as much as the arithmetic (a form with
// 4 % fewer FMA-pipe operations alone measured the same): the undecided nodes' tests
// run as one packed pair per lane, the box around the targets decides some of them, the
// push positions come from ballots instead of a shuffle scan, and the next round's
// records are prefetched before a batch.  Walk ms: 16,411 particles 0.218 -> 0.200,
// 200,003: 1.78 -> 1.69, 1M 8.24 -> 7.91, 4M 34.0 -> 33.1; strict 1M 11.45 -> 11.20; adjoint call
// of 100,003 particles 1.97 -> 1.90.
//
// kStrict (PEPCG_PRECISION_MIXED_STRICT): every interaction offset is the
// target minus the node centre formed in FP64 and then rounded, the FP32 sums
// of a batch are Kahan-compensated, and the group's MAC decisions equal the
// FP64 group walk's (k_walk_tile64 with two targets per lane): the bounding-
// sphere test is made conservative by a relative margin, and every node it
// leaves undecided gets the reference's FP64 test per target.  Twig records
// carry the FP64 node centre; four blocks per SM (128 registers).
template <bool kStrict>
__global__ void __launch_bounds__(kMixThreads, kStrict ? 4 : 5)
    k_walk_group64(MixArgs A, int* __restrict__ gstack) {
  using TwigRec = typename std::conditional<kStrict, StagedTwigS, StagedTwig>::type;
  __shared__ float s_bl2[kMaxLevel + 1];
  __shared__ double s_bl2d[kStrict ? kMaxLevel + 1 : 1];
  __shared__ double s_vb[3 * 125];
  __shared__ TwigRec s_tw[kWW][kRing];
  __shared__ StagedLeaf s_lf[kWW][kRing];
  // the two targets' FP64 sums (E, phi) live here rather than in registers: they
  // change once per batch of 32 records, and the registers go to the batches
  __shared__ double s_acc[8][kMixThreads];
  for (int i = threadIdx.x; i <= kMaxLevel; i += blockDim.x) {
    s_bl2[i] = (float)A.bl2[i];
    if constexpr (kStrict) s_bl2d[i] = A.bl2[i];
  }
  for (int i = threadIdx.x; i < 3 * A.nbox; i += blockDim.x) s_vb[i] = A.vbox[i];
  const uint32_t st = *A.tree_status;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  int* stack = gstack + (int64_t)(blockIdx.x * kWW + w) * kStackCap;
  TwigRec* stw = s_tw[w];
  StagedLeaf* stl = s_lf[w];
  const float theta2 = A.theta2;
  const int64_t nbuckets = st & ST_TIMEOUT ? 0 : (A.nt + 63) / 64;
  unsigned long long c_leaf = 0, c_twig = 0, c_mac = 0;
  for (;;) {
    unsigned b = 0;
    if (lane == 0) b = atomicAdd(A.queue, 1u);
    b = __shfl_sync(0xffffffffu, b, 0);
    if ((int64_t)b >= nbuckets) break;
    const int64_t t0 = (int64_t)b * 64;
    const int cnt = (int)min((int64_t)64, A.nt - t0);
    const bool v0 = lane < cnt, v1 = lane + 32 < cnt;
    const unsigned vm0 = __ballot_sync(0xffffffffu, v0), vm1 = __ballot_sync(0xffffffffu, v1);
    const int64_t ta = t0 + lane, tb = t0 + 32 + lane;
    double pxa = 0, pya = 0, pza = 0, pxb = 0, pyb = 0, pzb = 0;
    double &Ea0 = s_acc[0][threadIdx.x], &Ea1 = s_acc[1][threadIdx.x], &Ea2 = s_acc[2][threadIdx.x],
           &PHa = s_acc[3][threadIdx.x], &Eb0 = s_acc[4][threadIdx.x], &Eb1 = s_acc[5][threadIdx.x],
           &Eb2 = s_acc[6][threadIdx.x], &PHb = s_acc[7][threadIdx.x];
    double* acc = &s_acc[0][threadIdx.x];
    Ea0 = Ea1 = Ea2 = PHa = Eb0 = Eb1 = Eb2 = PHb = 0.0;
    double W = 0;  // interactions of this call (the same list for all targets)
    if (v0) {
      pxa = A.tx[ta]; pya = A.ty[ta]; pza = A.tz[ta];
      Ea0 = A.ex[ta]; Ea1 = A.ey[ta]; Ea2 = A.ez[ta]; PHa = A.pot[ta];
    }
    if (v1) {
      pxb = A.tx[tb]; pyb = A.ty[tb]; pzb = A.tz[tb];
      Eb0 = A.ex[tb]; Eb1 = A.ey[tb]; Eb2 = A.ez[tb]; PHb = A.pot[tb];
    }
    double lo[3] = {v0 ? pxa : INFINITY, v0 ? pya : INFINITY, v0 ? pza : INFINITY};
    double hi[3] = {v0 ? pxa : -INFINITY, v0 ? pya : -INFINITY, v0 ? pza : -INFINITY};
    if (v1) {
      lo[0] = fmin(lo[0], pxb); lo[1] = fmin(lo[1], pyb); lo[2] = fmin(lo[2], pzb);
      hi[0] = fmax(hi[0], pxb); hi[1] = fmax(hi[1], pyb); hi[2] = fmax(hi[2], pzb);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d)
      for (int o = 16; o > 0; o >>= 1) {
        lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
        hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
      }
    const double g0x = 0.5 * (lo[0] + hi[0]), g0y = 0.5 * (lo[1] + hi[1]), g0z = 0.5 * (lo[2] + hi[2]);
    const float rxa = (float)(pxa - g0x), rya = (float)(pya - g0y), rza = (float)(pza - g0z);
    const float rxb = (float)(pxb - g0x), ryb = (float)(pyb - g0y), rzb = (float)(pzb - g0z);
    float rg = fmaxf(v0 ? sqrtf(rxa * rxa + rya * rya + rza * rza) : 0.f,
                     v1 ? sqrtf(rxb * rxb + ryb * ryb + rzb * rzb) : 0.f);
    for (int o = 16; o > 0; o >>= 1) rg = fmaxf(rg, __shfl_xor_sync(0xffffffffu, rg, o));
    // the sphere and the box must contain every target after rounding
    rg = rg * 1.0001f + 1e-30f;
    const float hx = (float)(0.5 * (hi[0] - lo[0])) * 1.0001f + 1e-30f,
                hy = (float)(0.5 * (hi[1] - lo[1])) * 1.0001f + 1e-30f,
                hz = (float)(0.5 * (hi[2] - lo[2])) * 1.0001f + 1e-30f;
    bool complete = true;
    for (int ib = 0; ib < A.nbox; ++ib) {
      const double vx = s_vb[3 * ib], vy = s_vb[3 * ib + 1], vz = s_vb[3 * ib + 2];
      const double gx = g0x - vx, gy = g0y - vy, gz = g0z - vz;
      // the targets' shifted positions x - vbox (the strict form's offsets)
      const double sxa = pxa - vx, sya = pya - vy, sza = pza - vz;
      const double sxb = pxb - vx, syb = pyb - vy, szb = pzb - vz;
      const Targets64 T{rxa, rya, rza, rxb, ryb, rzb, sxa, sya, sza, sxb, syb, szb};
      int64_t partner = 0;
      int nT = 0, hT = 0, nL = 0, hL = 0;
      int top = 1;
      if (lane == 0) stack[0] = 0;
      __syncwarp();
      auto flush_twigs = [&](int n) {
        cp_async_wait_all();
        __syncwarp();
        if (v0) {
          twig_batch64<kStrict>(stw, hT, n, kRing, T, A.eps2, acc, kMixThreads);
          c_twig += (unsigned)n * (v1 ? 2u : 1u);
        }
        W += (double)n;
        hT = (hT + n) & (kRing - 1);
        nT -= n;
        __syncwarp();
      };
      auto flush_leaves = [&](int n) {
        __syncwarp();
        if (v0) {
          const unsigned nuse =
              leaf_batch64<kStrict>(stl, hL, n, kRing, T, v1, A, ta, tb,
                                    [&](const StagedLeaf&) { return make_double3(vx, vy, vz); },
                                    acc, kMixThreads);
          c_leaf += (unsigned)n * (v1 ? 2u : 1u) - nuse;
        }
        W += (double)n;
        hL = (hL + n) & (kRing - 1);
        nL -= n;
        __syncwarp();
      };
      while (top > 0) {
        const int take = top < 32 ? top : 32;
        top -= take;
        const int node = lane < take ? stack[top + lane] : -1;
        __syncwarp();
        bool isleaf = false, accept = false, open = false, amb = false;
        float cx = 0.f, cy = 0.f, cz = 0.f, bl = 0.f;
        double bld = 0.0;  // the strict form's FP64 MAC threshold
        double4 a = make_double4(0, 0, 0, 0);
        // the node's level-ordered record: centre and charge, then its links
        // (first child, level | leaf flag | child count, leaves, RPO index);
        // siblings are consecutive, so one round's loads are mostly runs
        int4 lk = make_int4(0, 0, 0, 0);
        if (node >= 0) {
          const LevelRecord* rec = A.drec + node;
          a = ld256(&rec->pos);
          lk = rec->link;
          cx = (float)(a.x - gx); cy = (float)(a.y - gy); cz = (float)(a.z - gz);
          if (lk.y & kLeafFlag) {
            isleaf = true;
          } else {
            bl = A.macb ? (float)A.macb[lk.w] : s_bl2[lk.y & 0xff];
            const float dc = sqrtf(cx * cx + cy * cy + cz * cz);
            float dmin = dc - rg, dmax = dc + rg;
            if constexpr (kStrict) {
              // conservative: the sphere decides only where the FP64 test of
              // every target certainly agrees
              bld = A.macb ? A.macb[lk.w] : s_bl2d[lk.y & 0xff];
              dmin = dc * (1.0f - 1e-5f) - rg;
              dmax = dc * (1.0f + 1e-5f) + rg;
            }
            if (dmin > 0.f && theta2 * (dmin * dmin) > bl) {
              accept = true;
              c_mac += 1;
            } else if (!(theta2 * (dmax * dmax) > bl)) {
              open = true;
              c_mac += 1;
            } else {
              amb = true;
            }
            if (amb) {
              // no target is nearer than their box: accepted without a test per
              // target (counted as one test each, as the tests below would)
              const float ax = fmaxf(fabsf(cx) - hx, 0.f), ay = fmaxf(fabsf(cy) - hy, 0.f),
                          az = fmaxf(fabsf(cz) - hz, 0.f);
              if (theta2 * ((ax * ax + ay * ay + az * az) * (1.0f - 1e-5f)) > bl) {
                amb = false;
                accept = true;
                c_mac += (unsigned)cnt;
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
            // the reference's operation order: theta2 * dist2 > boxlength2
            const double ux = __shfl_sync(0xffffffffu, a.x, j);
            const double uy = __shfl_sync(0xffffffffu, a.y, j);
            const double uz = __shfl_sync(0xffffffffu, a.z, j);
            const double ub = __shfl_sync(0xffffffffu, bld, j);
            double dx = sxa - ux, dy = sya - uy, dz = sza - uz;
            double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
            fa = v0 && !(__dmul_rn(A.theta2d, d2) > ub);
            dx = sxb - ux; dy = syb - uy; dz = szb - uz;
            d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
            fb = v1 && !(__dmul_rn(A.theta2d, d2) > ub);
          } else {
            const float ux = __shfl_sync(0xffffffffu, cx, j);
            const float uy = __shfl_sync(0xffffffffu, cy, j);
            const float uz = __shfl_sync(0xffffffffu, cz, j);
            const float ub = __shfl_sync(0xffffffffu, bl, j);
            const float2 dx = __fadd2_rn(make_float2(rxa, rxb), f2(-ux)),
                         dy = __fadd2_rn(make_float2(rya, ryb), f2(-uy)),
                         dz = __fadd2_rn(make_float2(rza, rzb), f2(-uz));
            const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
            fa = v0 && !(theta2 * d2.x > ub);
            fb = v1 && !(theta2 * d2.y > ub);
          }
          const unsigned f0 = __ballot_sync(0xffffffffu, fa);
          const unsigned f1 = __ballot_sync(0xffffffffu, fb);
          if (lane == j) {
            accept = (f0 | f1) == 0;
            open = !accept;
            // MAC evaluations up to the first failing target, in target order
            c_mac += (unsigned)(f0 ? __popc(vm0 & ((2u << (__ffs(f0) - 1)) - 1u))
                                   : __popc(vm0) + (f1 ? __popc(vm1 & ((2u << (__ffs(f1) - 1)) - 1u))
                                                       : __popc(vm1)));
          }
        }
        const unsigned lb = __ballot_sync(0xffffffffu, isleaf);
        const unsigned ab = __ballot_sync(0xffffffffu, accept);
        if (isleaf) {
          StagedLeaf& r = stl[(hL + nL + __popc(lb & lt)) & (kRing - 1)];
          r.c = make_float4(cx, cy, cz, (float)a.w);
          r.x = a.x; r.y = a.y; r.z = a.z;
          partner += 1;
        }
        if (accept) {
          TwigRec& r = stw[(hT + nT + __popc(ab & lt)) & (kRing - 1)];
          if constexpr (kStrict) {
            r.cx = a.x;
            r.cy = a.y;
            r.cz = a.z;
          } else {
            r.c = make_float4(-cx, -cy, -cz, (float)a.w);
          }
          const float4* m = A.mom32 + kMom32Stride * (int64_t)lk.w;
          cp_async16(&r.m0, m);
          cp_async16(&r.m1, m + 1);
          cp_async16(&r.m2, m + 2);
          partner += lk.z;
        }
        nL += __popc(lb);
        nT += __popc(ab);
        // an opened twig's children: level-order positions first .. first + nch - 1
        const int npush = open ? min(8, lk.y >> 16) : 0;
        int total;
        const int off = warp_excl_scan8(npush, lt, total);
        if (top + total > kStackCap) {
          complete = false;
          break;
        }
        if (npush > 0) {
          int* dst = stack + top + off;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < npush) dst[k] = lk.x + k;
        }
        top += total;
        __syncwarp();
        if (nT >= 32 || nL >= 32) {  // the next round's records come meanwhile
          const int nx = top < 32 ? top : 32;
          if (lane < nx)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(A.drec + stack[top - nx + lane]));
        }
        if (nT >= 32) flush_twigs(32);
        if (nL >= 32) flush_leaves(32);
      }
      if (nT > 0) flush_twigs(nT);
      if (nL > 0) flush_leaves(nL);
      for (int o = 16; o > 0; o >>= 1) partner += __shfl_xor_sync(0xffffffffu, partner, o);
      if (partner != A.npart) complete = false;
    }
    if (v0) {
      A.ex[ta] = Ea0; A.ey[ta] = Ea1; A.ez[ta] = Ea2; A.pot[ta] = PHa; A.work[ta] = A.work[ta] + W;
    }
    if (v1) {
      A.ex[tb] = Eb0; A.ey[tb] = Eb1; A.ez[tb] = Eb2; A.pot[tb] = PHb; A.work[tb] = A.work[tb] + W;
    }
    if (__any_sync(0xffffffffu, !complete) && lane == 0) atomicOr(A.status, ST_INCOMPLETE);
  }
  cp_async_wait_all();
  warp_add3(A.counters, c_leaf, c_twig, c_mac);
}

// Simple-walk semantics (module_tree_walk_simple.f90:256-385) with several
// reference tiles per warp and FP32 interactions: the whole tiles of one
// pack (at most 32 targets, k_pack_tiles) walk the tree together in forward
// preorder -- at each step the lanes whose tile stands at
// the smallest forward-preorder index evaluate that node, and each tile
// decides accept / open by a ballot over its own lanes (the MAC on the FP32
// offsets, target minus node centre formed in FP64).  Sums as in the
// per-target mixed walk: FP32 over chunks of kChunk steps, then FP64.
__global__ void __launch_bounds__(kMixThreads) k_walk_tilepack_mixed(MixArgs A) {
  __shared__ float s_bl2[kMaxLevel + 1];
  __shared__ double s_vb[3 * 125];
  for (int i = threadIdx.x; i <= kMaxLevel; i += blockDim.x) s_bl2[i] = (float)A.bl2[i];
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
    if ((int64_t)b >= npk) break;
    int tl0, len;
    const bool valid = pack_lane(A.pstart, A.tflag, b, lane, tl0, len);
    if (!__any_sync(0xffffffffu, valid)) {
      if (lane == 0) atomicOr(A.status, ST_INCOMPLETE);  // a pack must start with a tile
      continue;
    }
    const int64_t t = A.pstart[b] + lane;
    const unsigned tmask = valid ? (((len >= 32) ? 0xffffffffu : ((1u << len) - 1u)) << tl0) : 0u;
    double px = 0, py = 0, pz = 0, E0 = 0, E1 = 0, E2 = 0, PH = 0, W8 = 0;
    if (valid) {
      px = A.tx[t]; py = A.ty[t]; pz = A.tz[t];
      E0 = A.ex[t]; E1 = A.ey[t]; E2 = A.ez[t]; PH = A.pot[t]; W8 = A.work[t];
    }
    bool complete = true;
    for (int ib = 0; ib < A.nbox; ++ib) {
      const double sx = px - s_vb[3 * ib], sy = py - s_vb[3 * ib + 1], sz = pz - s_vb[3 * ib + 2];
      float ax = 0.f, ay = 0.f, az = 0.f, ap = 0.f;
      int steps = 0;
      unsigned u = 0, uf = 0;  // the root
      int64_t partner = 0;
      for (;;) {
        const unsigned f = __reduce_min_sync(0xffffffffu, valid ? uf : 0xffffffffu);
        if (f >= M) break;
        // the lanes at node f: whole tiles at the same node
        const unsigned am = __ballot_sync(0xffffffffu, valid && uf == f);
        if (valid && uf == f) {
          // one round of loads, the moments and leaf count included
          const double4 a = A.nc4[u];
          const int2 mu = A.meta[u];
          const int2 fw = A.fwd[u];
          const int2 ff = A.fwdf[u];
          const float4* mu4 = A.mom32 + kMom32Stride * (int64_t)u;
          const float4 m0 = mu4[0], m1 = mu4[1], m2 = mu4[2];
          const int nlv = A.nleaves[u];
          const double dx64 = sx - a.x, dy64 = sy - a.y, dz64 = sz - a.z;
          const float dx = (float)dx64, dy = (float)dy64, dz = (float)dz64;
          if (mu.y & kLeafFlag) {
            partner += 1;
            W8 += 1.0;
            if (!(dx64 == 0.0 && dy64 == 0.0 && dz64 == 0.0)) {
              leaf32((float)a.w, dx, dy, dz, A.eps2, ax, ay, az, ap);
              ++c_leaf;
            }
            u = (unsigned)fw.y;
            uf = (unsigned)ff.y;
          } else {
            const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            const bool ok = A.theta2 * r2 > (A.macb ? (float)A.macb[u] : s_bl2[mu.y & 0xff]);
            const unsigned tf = __ballot_sync(am, !ok) & tmask;
            // MAC evaluations stop at the tile's first failing target
            const int first_fail = tf ? __ffs(tf) - 1 : 32;
            if (lane <= first_fail) ++c_mac;
            if (tf == 0) {
              partner += nlv;
              twig32(m0, m1, m2, dx, dy, dz, A.eps2, ax, ay, az, ap);
              ++c_twig;
              W8 += 1.0;
              u = (unsigned)fw.y;
              uf = (unsigned)ff.y;
            } else {
              u = (unsigned)fw.x;
              uf = (unsigned)ff.x;
            }
          }
          if (++steps == kChunk) {
            E0 += (double)ax; E1 += (double)ay; E2 += (double)az; PH += (double)ap;
            ax = ay = az = ap = 0.f;
            steps = 0;
          }
        }
        __syncwarp();
      }
      E0 += (double)ax; E1 += (double)ay; E2 += (double)az; PH += (double)ap;
      if (valid && partner != A.npart) complete = false;
    }
    if (valid) {
      A.ex[t] = E0; A.ey[t] = E1; A.ez[t] = E2; A.pot[t] = PH; A.work[t] = W8;
    }
    if (__any_sync(0xffffffffu, !complete) && lane == 0) atomicOr(A.status, ST_INCOMPLETE);
  }
  warp_add3(A.counters, c_leaf, c_twig, c_mac);
}

// per-target semantics (module_tree_walk_pthreads.f90:558-765) with FP32
// interactions; the MAC is evaluated on the FP32 offsets
__global__ void __launch_bounds__(kMixThreads) k_walk_target_mixed(MixArgs A) {
  __shared__ float s_bl2[kMaxLevel + 1];
  __shared__ double s_vb[3 * 125];
  for (int i = threadIdx.x; i <= kMaxLevel; i += blockDim.x) s_bl2[i] = (float)A.bl2[i];
  for (int i = threadIdx.x; i < 3 * A.nbox; i += blockDim.x) s_vb[i] = A.vbox[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const unsigned M = (unsigned)A.M;
  unsigned long long c_leaf = 0, c_twig = 0, c_mac = 0;
  for (;;) {
    unsigned b = 0;
    if (lane == 0) b = atomicAdd(A.queue, 1u);
    b = __shfl_sync(0xffffffffu, b, 0);
    if ((int64_t)b * 32 >= A.nt) break;
    const int64_t t = (int64_t)b * 32 + lane;
    const bool valid = t < A.nt;
    double px = 0, py = 0, pz = 0, E0 = 0, E1 = 0, E2 = 0, PH = 0, W = 0;
    if (valid) {
      px = A.tx[t]; py = A.ty[t]; pz = A.tz[t];
      E0 = A.ex[t]; E1 = A.ey[t]; E2 = A.ez[t]; PH = A.pot[t]; W = A.work[t];
    }
    bool complete = true;
    for (int ib = 0; ib < A.nbox; ++ib) {
      const double sx = px - s_vb[3 * ib], sy = py - s_vb[3 * ib + 1], sz = pz - s_vb[3 * ib + 2];
      float ax = 0.f, ay = 0.f, az = 0.f, ap = 0.f;
      int steps = 0;
      unsigned next = valid ? 1u : M;
      int64_t partner = 0;
      for (;;) {
        const unsigned u = __reduce_min_sync(0xffffffffu, next);
        if (u >= M) break;
        if (next == u) {
          // one round of loads: the moments and leaf count are requested with
          // the centre, before the MAC decides whether they are used
          const double4 a = A.nc4[u];
          const int2 mu = A.meta[u];
          const float4* mu4 = A.mom32 + kMom32Stride * (int64_t)u;
          const float4 m0 = mu4[0], m1 = mu4[1], m2 = mu4[2];
          const int nlv = A.nleaves[u];
          const double dx64 = sx - a.x, dy64 = sy - a.y, dz64 = sz - a.z;
          const float dx = (float)dx64, dy = (float)dy64, dz = (float)dz64;
          if (mu.y & kLeafFlag) {
            partner += 1;
            W += 1.0;
            if (!(dx64 == 0.0 && dy64 == 0.0 && dz64 == 0.0)) {
              leaf32((float)a.w, dx, dy, dz, A.eps2, ax, ay, az, ap);
              ++c_leaf;
            }
            next = u + 1;
          } else {
            ++c_mac;
            const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            if (A.theta2 * r2 > (A.macb ? (float)A.macb[u] : s_bl2[mu.y & 0xff])) {
              partner += nlv;
              twig32(m0, m1, m2, dx, dy, dz, A.eps2, ax, ay, az, ap);
              ++c_twig;
              W += 1.0;
              next = (unsigned)mu.x;
            } else {
              next = u + 1;
            }
          }
          if (++steps == kChunk) {
            E0 += (double)ax; E1 += (double)ay; E2 += (double)az; PH += (double)ap;
            ax = ay = az = ap = 0.f;
            steps = 0;
          }
        }
      }
      E0 += (double)ax; E1 += (double)ay; E2 += (double)az; PH += (double)ap;
      if (valid && partner != A.npart) complete = false;
    }
    if (valid) {
      A.ex[t] = E0; A.ey[t] = E1; A.ez[t] = E2; A.pot[t] = PH; A.work[t] = W;
    }
    if (__any_sync(0xffffffffu, !complete) && lane == 0) atomicOr(A.status, ST_INCOMPLETE);
  }
  warp_add3(A.counters, c_leaf, c_twig, c_mac);
}

// ---------------------------------------------------------------------------
// Adjoint of the mixed group walk with 64-target buckets.  The traversal, the
// FP32 group-centred MAC and the staging are k_walk_group64's, so each
// bucket's interaction list is the forward list.  The staged batches are
// evaluated transposed: lane j takes node record j of the batch and loops over
// the bucket's 64 targets, whose group-centred FP32 offsets and gradients are
// broadcast from shared memory two at a time (one packed FP32 operation per
// target pair).  A lane thus sums its node's adjoint record over the bucket
// without any cross-lane reduction, in FP32 as the forward sums its batches,
// and adds it to the node's FP64 record with one atomic per value.  The terms
// are the transposes of the forward's (the FP64 forms and their derivation
// are in adjoint.cu, twig_adj / leaf_adj), rewritten with T = 3M, v = T d and
// dTd = d.v: with s1 = gphi R1 and s3 = 3 gphi R2,
//   qbar   += gphi R0                      (+ (g.d) R1)
//   pbar   -= s1 d                         (+ R1 g - 3 (g.d) R2 d)
//   Qbar_kl += s3 d_k d_l - delta_kl s1    (+ 15 (g.d) R3 d_k d_l - 3 R2 (g_k d_l + g_l d_k + delta_kl g.d))
//   cocbar += gphi [ce d + R1 p - 2 R2 v]  (+ the Hessian terms of twig_adj)
// with ce = q R1 - 3 R2 (p.d + tr) + 5 R3 dTd; sums over the targets of a
// node-constant factor (the p terms, the delta terms) are taken once per batch.
// ---------------------------------------------------------------------------
// Four resident blocks per SM (128 registers, the twig terms' pair
// accumulators and node constants stay in registers): at 4M the full
// gradient takes 88 ms against 111 ms at five blocks (96 registers, spills).
template <bool kWithE>
__global__ void __launch_bounds__(kMixThreads, 4)
    k_adj_group64(AdjMixArgs A, int* __restrict__ gstack) {
  __shared__ float s_bl2[kMaxLevel + 1];
  __shared__ double s_vb[3 * 125];
  __shared__ StagedTwig s_tw[kWW][kRing];
  __shared__ StagedLeafA s_lf[kWW][kRing];
  // per warp and target pair p (targets t0 + p, t0 + 32 + p): (rx, rx', ry, ry'),
  // (rz, rz', gphi, gphi'), (gx, gx', gy, gy'), (gz, gz', -, -)
  __shared__ float4 s_tg[kWW][32][kWithE ? 4 : 2];
  for (int i = threadIdx.x; i <= kMaxLevel; i += blockDim.x) s_bl2[i] = (float)A.bl2[i];
  for (int i = threadIdx.x; i < 3 * A.nbox; i += blockDim.x) s_vb[i] = A.vbox[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  int* stack = gstack + (int64_t)(blockIdx.x * kWW + w) * kStackCap;
  StagedTwig* stw = s_tw[w];
  StagedLeafA* stl = s_lf[w];
  float4(*tg)[kWithE ? 4 : 2] = s_tg[w];
  const float theta2 = A.theta2;
  const float2 E2 = f2(A.eps2);
  const int64_t nbuckets = (A.nt + 63) / 64;
  unsigned long long c_leaf = 0, c_twig = 0, c_mac = 0;
  for (;;) {
    unsigned b = 0;
    if (lane == 0) b = atomicAdd(A.queue, 1u);
    b = __shfl_sync(0xffffffffu, b, 0);
    if ((int64_t)b >= nbuckets) break;
    const int64_t t0 = (int64_t)b * 64;
    const int cnt = (int)min((int64_t)64, A.nt - t0);
    const bool v0 = lane < cnt, v1 = lane + 32 < cnt;
    const unsigned vm0 = __ballot_sync(0xffffffffu, v0), vm1 = __ballot_sync(0xffffffffu, v1);
    const int nvalid = __popc(vm0) + __popc(vm1);
    const int64_t ta = t0 + lane, tb = t0 + 32 + lane;
    double pxa = 0, pya = 0, pza = 0, pxb = 0, pyb = 0, pzb = 0;
    float gpa = 0.f, gpb = 0.f, gxa = 0.f, gya = 0.f, gza = 0.f, gxb = 0.f, gyb = 0.f, gzb = 0.f;
    if (v0) {
      pxa = A.tx[ta]; pya = A.ty[ta]; pza = A.tz[ta];
      gpa = (float)A.gphi[ta];
      if (kWithE) { gxa = (float)A.gex[ta]; gya = (float)A.gey[ta]; gza = (float)A.gez[ta]; }
    }
    if (v1) {
      pxb = A.tx[tb]; pyb = A.ty[tb]; pzb = A.tz[tb];
      gpb = (float)A.gphi[tb];
      if (kWithE) { gxb = (float)A.gex[tb]; gyb = (float)A.gey[tb]; gzb = (float)A.gez[tb]; }
    }
    double lo[3] = {v0 ? pxa : INFINITY, v0 ? pya : INFINITY, v0 ? pza : INFINITY};
    double hi[3] = {v0 ? pxa : -INFINITY, v0 ? pya : -INFINITY, v0 ? pza : -INFINITY};
    if (v1) {
      lo[0] = fmin(lo[0], pxb); lo[1] = fmin(lo[1], pyb); lo[2] = fmin(lo[2], pzb);
      hi[0] = fmax(hi[0], pxb); hi[1] = fmax(hi[1], pyb); hi[2] = fmax(hi[2], pzb);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d)
      for (int o = 16; o > 0; o >>= 1) {
        lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
        hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
      }
    const double g0x = 0.5 * (lo[0] + hi[0]), g0y = 0.5 * (lo[1] + hi[1]), g0z = 0.5 * (lo[2] + hi[2]);
    const float rxa = (float)(pxa - g0x), rya = (float)(pya - g0y), rza = (float)(pza - g0z);
    const float rxb = (float)(pxb - g0x), ryb = (float)(pyb - g0y), rzb = (float)(pzb - g0z);
    float rg = fmaxf(v0 ? sqrtf(rxa * rxa + rya * rya + rza * rza) : 0.f,
                     v1 ? sqrtf(rxb * rxb + ryb * ryb + rzb * rzb) : 0.f);
    for (int o = 16; o > 0; o >>= 1) rg = fmaxf(rg, __shfl_xor_sync(0xffffffffu, rg, o));
    // the sphere and the box must contain every target after rounding
    rg = rg * 1.0001f + 1e-30f;
    const float hx = (float)(0.5 * (hi[0] - lo[0])) * 1.0001f + 1e-30f,
                hy = (float)(0.5 * (hi[1] - lo[1])) * 1.0001f + 1e-30f,
                hz = (float)(0.5 * (hi[2] - lo[2])) * 1.0001f + 1e-30f;
    // an absent target sits far away with zero gradients: it adds exact zeros
    tg[lane][0] = make_float4(v0 ? rxa : 1e10f, v1 ? rxb : 1e10f, v0 ? rya : 1e10f, v1 ? ryb : 1e10f);
    tg[lane][1] = make_float4(v0 ? rza : 1e10f, v1 ? rzb : 1e10f, gpa, gpb);
    if constexpr (kWithE) {
      tg[lane][2] = make_float4(gxa, gxb, gya, gyb);
      tg[lane][3] = make_float4(gza, gzb, 0.f, 0.f);
    }
    __syncwarp();
    bool complete = true;
    for (int ib = 0; ib < A.nbox; ++ib) {
      const double vx = s_vb[3 * ib], vy = s_vb[3 * ib + 1], vz = s_vb[3 * ib + 2];
      const double gx = g0x - vx, gy = g0y - vy, gz = g0z - vz;
      int64_t partner = 0;
      int nT = 0, hT = 0, nL = 0, hL = 0;
      int top = 1;
      if (lane == 0) stack[0] = 0;
      __syncwarp();
      // twig records: lane j sums node j's record over the bucket's targets
      auto flush_twigs = [&](int n) {
        cp_async_wait_all();
        __syncwarp();
        if (lane < n)
          adj_twig_record<kWithE>(stw[(hT + lane) & (kRing - 1)], tg, E2, A.adj);
        c_twig += (unsigned)n * (unsigned)nvalid;
        hT = (hT + n) & (kRing - 1);
        nT -= n;
        __syncwarp();
      };
      // leaf records: qbar += gphi R0 (+ g.d R1), cocbar += q [(gphi R1 (+ 3 g.d R2)) d (- R1 g)]
      auto flush_leaves = [&](int n) {
        __syncwarp();
        if (lane < n)
          adj_leaf_record<kWithE>(stl[(hL + lane) & (kRing - 1)], tg, E2, A, t0,
                                  make_double3(vx, vy, vz));
        c_leaf += (unsigned)n * (unsigned)nvalid;
        hL = (hL + n) & (kRing - 1);
        nL -= n;
        __syncwarp();
      };
      // the traversal and MAC of k_walk_group64 (same decisions, same lists)
      while (top > 0) {
        const int take = top < 32 ? top : 32;
        top -= take;
        const int node = lane < take ? stack[top + lane] : -1;
        __syncwarp();
        bool isleaf = false, accept = false, open = false, amb = false;
        float cx = 0.f, cy = 0.f, cz = 0.f, bl = 0.f;
        double4 a = make_double4(0, 0, 0, 0);
        // the node's level-ordered record and links (k_walk_group64's traversal);
        // the adjoint records are in the same level order
        int4 lk = make_int4(0, 0, 0, 0);
        if (node >= 0) {
          const LevelRecord* rec = A.drec + node;
          a = ld256(&rec->pos);
          lk = rec->link;
          cx = (float)(a.x - gx); cy = (float)(a.y - gy); cz = (float)(a.z - gz);
          if (lk.y & kLeafFlag) {
            isleaf = true;
          } else {
            bl = A.macb ? (float)A.macb[lk.w] : s_bl2[lk.y & 0xff];
            const float dc = sqrtf(cx * cx + cy * cy + cz * cz);
            const float dmin = dc - rg, dmax = dc + rg;
            if (dmin > 0.f && theta2 * (dmin * dmin) > bl) {
              accept = true;
              c_mac += 1;
            } else if (!(theta2 * (dmax * dmax) > bl)) {
              open = true;
              c_mac += 1;
            } else {
              amb = true;
            }
            if (amb) {
              // no target is nearer than their box: accepted without a test per
              // target (counted as one test each, as the tests below would)
              const float ax = fmaxf(fabsf(cx) - hx, 0.f), ay = fmaxf(fabsf(cy) - hy, 0.f),
                          az = fmaxf(fabsf(cz) - hz, 0.f);
              if (theta2 * ((ax * ax + ay * ay + az * az) * (1.0f - 1e-5f)) > bl) {
                amb = false;
                accept = true;
                c_mac += (unsigned)cnt;
              }
            }
          }
        }
        unsigned am = __ballot_sync(0xffffffffu, amb);
        while (am) {
          const int j = __ffs(am) - 1;
          am &= am - 1;
          const float ux = __shfl_sync(0xffffffffu, cx, j);
          const float uy = __shfl_sync(0xffffffffu, cy, j);
          const float uz = __shfl_sync(0xffffffffu, cz, j);
          const float ub = __shfl_sync(0xffffffffu, bl, j);
          const float2 dx = __fadd2_rn(make_float2(rxa, rxb), f2(-ux)),
                       dy = __fadd2_rn(make_float2(rya, ryb), f2(-uy)),
                       dz = __fadd2_rn(make_float2(rza, rzb), f2(-uz));
          const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
          const bool fa = v0 && !(theta2 * d2.x > ub);
          const bool fb = v1 && !(theta2 * d2.y > ub);
          const unsigned f0 = __ballot_sync(0xffffffffu, fa);
          const unsigned f1 = __ballot_sync(0xffffffffu, fb);
          if (lane == j) {
            accept = (f0 | f1) == 0;
            open = !accept;
            c_mac += (unsigned)(f0 ? __popc(vm0 & ((2u << (__ffs(f0) - 1)) - 1u))
                                   : __popc(vm0) + (f1 ? __popc(vm1 & ((2u << (__ffs(f1) - 1)) - 1u))
                                                       : __popc(vm1)));
          }
        }
        const unsigned lb = __ballot_sync(0xffffffffu, isleaf);
        const unsigned ab = __ballot_sync(0xffffffffu, accept);
        if (isleaf) {
          StagedLeafA& r = stl[(hL + nL + __popc(lb & lt)) & (kRing - 1)];
          r.c = make_float4(cx, cy, cz, (float)a.w);
          r.x = a.x; r.y = a.y; r.z = a.z;
          r.node = node;
          partner += 1;
        }
        if (accept) {
          StagedTwig& r = stw[(hT + nT + __popc(ab & lt)) & (kRing - 1)];
          r.c = make_float4(-cx, -cy, -cz, __int_as_float(node));
          const float4* m = A.mom32 + kMom32Stride * (int64_t)lk.w;
          cp_async16(&r.m0, m);
          cp_async16(&r.m1, m + 1);
          cp_async16(&r.m2, m + 2);
          partner += lk.z;
        }
        nL += __popc(lb);
        nT += __popc(ab);
        const int npush = open ? min(8, lk.y >> 16) : 0;
        int total;
        const int off = warp_excl_scan8(npush, lt, total);
        if (top + total > kStackCap) {
          complete = false;
          break;
        }
        if (npush > 0) {
          int* dst = stack + top + off;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < npush) dst[k] = lk.x + k;
        }
        top += total;
        __syncwarp();
        if (nT >= 32 || nL >= 32) {  // the next round's records come meanwhile
          const int nx = top < 32 ? top : 32;
          if (lane < nx)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(A.drec + stack[top - nx + lane]));
        }
        if (nT >= 32) flush_twigs(32);
        if (nL >= 32) flush_leaves(32);
      }
      if (nT > 0) flush_twigs(nT);
      if (nL > 0) flush_leaves(nL);
      for (int o = 16; o > 0; o >>= 1) partner += __shfl_xor_sync(0xffffffffu, partner, o);
      if (partner != A.npart) complete = false;
    }
    __syncwarp();
    if (__any_sync(0xffffffffu, !complete) && lane == 0) atomicOr(A.status, ST_INCOMPLETE);
  }
  cp_async_wait_all();
  warp_add3(A.counters, c_leaf, c_twig, c_mac);
}

}  // namespace

int launch_walk_mixed(Ctx* c, int64_t nt, const double* tx, const double* ty, const double* tz,
                      double* ex, double* ey, double* ez, double* pot, double* work,
                      const int2* tiles, int64_t ntiles, bool per_target,
                      const int32_t* tflag, const int32_t* pstart, const int32_t* npacks,
                      cudaStream_t s, int slot, int64_t shape_nt, bool keyed) {
  MixArgs A;
  A.nt = nt;
  A.tx = tx; A.ty = ty; A.tz = tz;
  A.nc4 = c->nc4.p;
  A.meta = c->meta.p;
  A.mom32 = reinterpret_cast<const float4*>(c->mom32.p);
  A.nleaves = c->nleaves.p;
  A.drec = c->drec.p;
  A.bl2 = c->d_box + 9;
  {
    int rc = prepare_mac(c, &A.macb);
    if (rc) return rc;
  }
  A.vbox = c->d_vbox;
  A.nbox = c->nboxes;
  A.theta2 = (float)c->prm.theta2;
  A.theta2d = c->prm.theta2;
  A.eps2 = (float)c->prm.eps2;
  A.M = (int32_t)c->nnodes;
  A.npart = c->n;
  A.ex = ex; A.ey = ey; A.ez = ez; A.pot = pot; A.work = work;
  A.counters = c->counters;
  A.status = c->d_status;
  A.queue = c->walk_queue(slot);
  A.tiles = tiles;
  A.ntiles = ntiles;
  A.fwd = c->fwd.p;
  A.fwdf = c->fwdf.p;
  A.tflag = tflag;
  A.pstart = pstart;
  A.npacks = npacks;
  A.tree_status = c->d_tree_status;
  BlockShape sh;
  const bool group64 = !per_target && !tflag && tiles == nullptr && c->group_size() == 64;
  const bool strict = c->prm.precision == PEPCG_PRECISION_MIXED_STRICT;
  if (group64 && block_walk_shape(shape_nt, c->n, strict ? BlockWalk::kStrict : BlockWalk::kDefault, keyed, &sh)) {
    const size_t per = (size_t)148 * 5 * kWW * kStackCap;
    if (!ensure(c, c->wstack, 2 * per, "walk stacks")) return PEPCG_ERR_OOM;
    if (launch_walk_block64(c, A, sh, strict, c->wstack.p + slot * per, s)) return PEPCG_OK;
  }
  COUNT_LAUNCH();
  if (per_target) {
    k_walk_target_mixed<<<148 * 8, kMixThreads, 0, s>>>(A);
  } else if (tflag) {
    k_walk_tilepack_mixed<<<148 * 8, kMixThreads, 0, s>>>(A);
  } else {
    // 5 resident blocks per SM (launch bounds: at most 96 registers; the
    // 64-target walk holds 39 KB of shared memory per block); the grid is
    // exactly one wave.  One set of stacks per walk stream.
    const int gblocks = 148 * 5;
    const size_t per = (size_t)gblocks * kWW * kStackCap;
    if (!ensure(c, c->wstack, 2 * per, "walk stacks")) return PEPCG_ERR_OOM;
    if (c->prm.precision == PEPCG_PRECISION_MIXED_STRICT)  // 4 blocks per SM
      k_walk_group64<true><<<148 * 4, kMixThreads, 0, s>>>(A, c->wstack.p + slot * per);
    else if (tiles == nullptr && c->group_size() == 64)
      k_walk_group64<false><<<gblocks, kMixThreads, 0, s>>>(A, c->wstack.p + slot * per);
    else
      k_walk_group_wide<<<gblocks, kMixThreads, 0, s>>>(A, c->wstack.p + slot * per, c->child8.p,
                                                        c->nchild.p);
  }
  return cuda_ok(c, cudaGetLastError(), "mixed walk launch") ? PEPCG_OK : PEPCG_ERR_CUDA;
}

// The adjoint walk of the mixed group walk with 64-target buckets: fills the
// twigs' and leaves' adjoint records (adj, 16 doubles per node, zeroed by the
// caller); the downward pass and the output are adjoint.cu's.
int launch_adjoint_group64(Ctx* c, int64_t nt, const double* tx, const double* ty,
                           const double* tz, const double* gex, const double* gey,
                           const double* gez, const double* gphi, bool with_e, cudaStream_t s) {
  if (nt == 0) return PEPCG_OK;  // no records; a grid of no blocks is refused
  AdjMixArgs A;
  A.nt = nt;
  A.tx = tx; A.ty = ty; A.tz = tz;
  A.gex = gex; A.gey = gey; A.gez = gez; A.gphi = gphi;
  A.nc4 = c->nc4.p;
  A.meta = c->meta.p;
  A.mom32 = reinterpret_cast<const float4*>(c->mom32.p);
  A.nleaves = c->nleaves.p;
  A.drec = c->drec.p;
  A.bl2 = c->d_box + 9;
  {
    int rc = prepare_mac(c, &A.macb);
    if (rc) return rc;
  }
  A.vbox = c->d_vbox;
  A.nbox = c->nboxes;
  A.theta2 = (float)c->prm.theta2;
  A.eps2 = (float)c->prm.eps2;
  A.npart = c->n;
  A.adj = c->adj.p;
  A.counters = c->counters;
  A.status = c->d_adj_status;
  A.queue = c->walk_queue();
  const int gblocks = 148 * 4;
  const size_t per = (size_t)gblocks * kWW * kStackCap;
  if (!ensure(c, c->wstack, 2 * per, "walk stacks")) return PEPCG_ERR_OOM;
  BlockShape sh;
  if (block_walk_shape(nt, c->n, BlockWalk::kAdjoint, false, &sh) &&
      launch_adj_block64(c, A, sh, with_e, c->wstack.p, s))
    return PEPCG_OK;
  COUNT_LAUNCH();
  if (with_e)
    k_adj_group64<true><<<gblocks, kMixThreads, 0, s>>>(A, c->wstack.p);
  else
    k_adj_group64<false><<<gblocks, kMixThreads, 0, s>>>(A, c->wstack.p);
  return cuda_ok(c, cudaGetLastError(), "mixed adjoint launch") ? PEPCG_OK : PEPCG_ERR_CUDA;
}

}  // namespace pepcg
