// mixed.cuh -- what the mixed-precision walks share (walk_mixed.cu, walk_block.cu):
// kernel arguments, the FP32 interactions, staging records, and the batches
// that the 64-target group walk and its adjoint evaluate from shared memory.
#pragma once

#include <type_traits>

#include "internal.cuh"

namespace pepcg {

constexpr int kMixThreads = 128;
constexpr int kChunk = 32;

struct MixArgs {
  int64_t nt;
  const double* tx;
  const double* ty;
  const double* tz;
  const double4* nc4;
  const int2* meta;
  const float4* mom32;  // kMom32Stride float4 per node, the first 3 used
  const int32_t* nleaves;
  const LevelRecord* drec;  // level-ordered node records with walk links (grow.cu)
  const double* bl2;
  const double* macb;  // per-twig MAC threshold, or nullptr: bl2 of the level (Barnes-Hut)
  const double* vbox;
  int nbox;
  float theta2;
  float eps2;
  double theta2d;  // theta2 in FP64 (the strict form's exact MAC)
  int32_t M;
  int64_t npart;
  double* ex;
  double* ey;
  double* ez;
  double* pot;
  double* work;
  unsigned long long* counters;
  uint32_t* status;
  unsigned int* queue;  // bucket counter, zeroed before the launch
  const int2* tiles;  // PER_TILE tiles, or nullptr for GROUP (implicit 32-target buckets)
  int64_t ntiles;
  // packed per-tile walk
  const int2* fwd;       // (first child, next after the subtree), RPO indices
  const int2* fwdf;      // the same as forward-preorder indices
  const int32_t* tflag;  // per target: length of the tile starting there, else 0
  const int32_t* pstart;  // packed per-tile walk: first target of each pack, then nt
  const int32_t* npacks;  // the number of packs (device)
  const uint32_t* tree_status;  // set: drec was not built
};

// 1/sqrt(x) by the PTX instruction rsqrt.approx.ftz.f32 (relative error below
// 2^-22, subnormal inputs and results flushed to zero).  The arguments here are
// squared distances plus eps2; a zero argument gives +inf and is selected away
// by the callers that can meet it (the leaves' self pairs).  rsqrtf would add a
// range fix-up for subnormal arguments on every call: at 4M this form takes the
// benchmark's walk from 38.5 to 36.0 ms with identical results.
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void leaf32(float q, float dx, float dy, float dz, float eps2,
                                       float& ax, float& ay, float& az, float& ap) {
  const float r2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps2)));
  const float ri = rsqrt_ftz(r2);
  const float qr = q * ri;
  const float qr3 = qr * ri * ri;
  ap += qr;
  ax = fmaf(qr3, dx, ax);
  ay = fmaf(qr3, dy, ay);
  az = fmaf(qr3, dz, az);
}

// m0 = (px, py, pz, 3qxx), m1 = (3qyy, 3qzz, 1.5qxy, 1.5qyz), m2 = (1.5qzx, tr, q, -),
// i.e. 3M with M the quadrupole matrix with halved off-diagonals; with
// A = d.p + tr, v = 3M d and B = d.v, in Horner form in 1/r^2:
//   phi += (q + (B/r^2 - A)/r^2) / r
//   E   += [d (q + (5B/r^2 - 3A)/r^2) + p - 2 v/r^2] / r^3
// where 5B/r^2 - 3A = 5 (B/r^2 - A) + 2A reuses the potential's inner term:
// 39 FP32 operations and one rsqrt per interaction.
__device__ __forceinline__ void twig32(float4 m0, float4 m1, float4 m2, float dx, float dy,
                                       float dz, float eps2, float& ax, float& ay, float& az,
                                       float& ap) {
  const float r2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps2)));
  const float ri = rsqrt_ftz(r2);
  const float ri2 = ri * ri;
  const float rd3 = ri * ri2;
  const float q = m2.z;
  const float A = fmaf(dx, m0.x, fmaf(dy, m0.y, fmaf(dz, m0.z, m2.y)));
  const float vx = fmaf(m0.w, dx, fmaf(m1.z, dy, m2.x * dz));
  const float vy = fmaf(m1.z, dx, fmaf(m1.x, dy, m1.w * dz));
  const float vz = fmaf(m2.x, dx, fmaf(m1.w, dy, m1.y * dz));
  const float B = fmaf(dx, vx, fmaf(dy, vy, dz * vz));
  const float t1 = fmaf(ri2, B, -A);
  ap = fmaf(ri, fmaf(ri2, t1, q), ap);
  const float t4 = fmaf(ri2, fmaf(5.0f, t1, A + A), q);
  const float m2r = -2.0f * ri2;
  ax = fmaf(rd3, fmaf(t4, dx, fmaf(m2r, vx, m0.x)), ax);
  ay = fmaf(rd3, fmaf(t4, dy, fmaf(m2r, vy, m0.y)), ay);
  az = fmaf(rd3, fmaf(t4, dz, fmaf(m2r, vz, m0.z)), az);
}

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }

// -a by the sign bits (integer operations: the FMA pipe is the busy one)
__device__ __forceinline__ float2 neg2(float2 a) {
  return make_float2(__uint_as_float(__float_as_uint(a.x) ^ 0x80000000u),
                     __uint_as_float(__float_as_uint(a.y) ^ 0x80000000u));
}

// twig32's interaction for two targets against the same node in packed FP32
// (sm_100 FFMA2 / FMUL2 / FADD2): each operation evaluates both targets' terms, and
// the node's moments enter as (m, m) pairs.  With s1 = A - B/r^2 and s2 = s1 - B/r^2,
//   phi = (q - s1/r^2) / r,   5B/r^2 - 3A = -(s1 + 2 s2),
// so E's coefficient of d follows from phi's inner term g = q - s1/r^2 as
// g - 2 s2/r^2: one operation less than twig32's form.
struct Twig2 {
  float2 ri, rd3, g, ex, ey, ez;  // phi = ri g, E = rd3 e
};
__device__ __forceinline__ Twig2 twig32x2_parts(float4 m0, float4 m1, float4 m2, float2 dx,
                                                float2 dy, float2 dz, float2 eps2) {
  const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, eps2)));
  const float2 ri = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
  const float2 ri2 = __fmul2_rn(ri, ri);
  const float2 n2 = neg2(ri2);
  const float2 m2r = __fmul2_rn(f2(-2.0f), ri2);
  const float2 A = __ffma2_rn(dx, f2(m0.x), __ffma2_rn(dy, f2(m0.y), __ffma2_rn(dz, f2(m0.z), f2(m2.y))));
  const float2 vx = __ffma2_rn(f2(m0.w), dx, __ffma2_rn(f2(m1.z), dy, __fmul2_rn(f2(m2.x), dz)));
  const float2 vy = __ffma2_rn(f2(m1.z), dx, __ffma2_rn(f2(m1.x), dy, __fmul2_rn(f2(m1.w), dz)));
  const float2 vz = __ffma2_rn(f2(m2.x), dx, __ffma2_rn(f2(m1.w), dy, __fmul2_rn(f2(m1.y), dz)));
  const float2 B = __ffma2_rn(dx, vx, __ffma2_rn(dy, vy, __fmul2_rn(dz, vz)));
  const float2 s1 = __ffma2_rn(n2, B, A);
  const float2 g = __ffma2_rn(n2, s1, f2(m2.z));
  const float2 t4 = __ffma2_rn(m2r, __ffma2_rn(n2, B, s1), g);
  Twig2 t;
  t.ri = ri;
  t.rd3 = __fmul2_rn(ri, ri2);
  t.g = g;
  t.ex = __ffma2_rn(t4, dx, __ffma2_rn(m2r, vx, f2(m0.x)));
  t.ey = __ffma2_rn(t4, dy, __ffma2_rn(m2r, vy, f2(m0.y)));
  t.ez = __ffma2_rn(t4, dz, __ffma2_rn(m2r, vz, f2(m0.z)));
  return t;
}

__device__ __forceinline__ void twig32x2(float4 m0, float4 m1, float4 m2, float2 dx, float2 dy,
                                         float2 dz, float2 eps2, float2& ax, float2& ay,
                                         float2& az, float2& ap) {
  const Twig2 t = twig32x2_parts(m0, m1, m2, dx, dy, dz, eps2);
  ap = __ffma2_rn(t.ri, t.g, ap);
  ax = __ffma2_rn(t.rd3, t.ex, ax);
  ay = __ffma2_rn(t.rd3, t.ey, ay);
  az = __ffma2_rn(t.rd3, t.ez, az);
}

// the terms of one interaction, returned instead of accumulated (the strict form
// adds them with compensation)
__device__ __forceinline__ void twig32x2_terms(float4 m0, float4 m1, float4 m2, float2 dx,
                                               float2 dy, float2 dz, float2 eps2, float2& ax,
                                               float2& ay, float2& az, float2& ap) {
  const Twig2 t = twig32x2_parts(m0, m1, m2, dx, dy, dz, eps2);
  ap = __fmul2_rn(t.ri, t.g);
  ax = __fmul2_rn(t.rd3, t.ex);
  ay = __fmul2_rn(t.rd3, t.ey);
  az = __fmul2_rn(t.rd3, t.ez);
}

// Kahan (compensated) summation, both lanes of a pair: s += v with the
// running compensation c (the sum is s - c)
__device__ __forceinline__ void kahan2(float2& s, float2& c, float2 v) {
  const float2 y = __fadd2_rn(v, make_float2(-c.x, -c.y));
  const float2 t = __fadd2_rn(s, y);
  c = __fadd2_rn(__fadd2_rn(t, make_float2(-s.x, -s.y)), make_float2(-y.x, -y.y));
  s = t;
}

__device__ __forceinline__ void warp_add3(unsigned long long* ctr, unsigned long long a,
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

constexpr int kStackCap = 8192;
constexpr int kWW = kMixThreads / 32;  // warps per block
constexpr int kRing = 64;              // staging ring (<= 31 pending + 32 new)

__device__ __forceinline__ int warp_excl_scan(int v, int lane, int& total) {
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  total = __shfl_sync(0xffffffffu, x, 31);
  return x - v;
}

// exclusive prefix of v in 0 .. 8 over the warp, from one ballot per bit
__device__ __forceinline__ int warp_excl_scan8(int v, unsigned lt, int& total) {
  int off = 0;
  total = 0;
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const unsigned m = __ballot_sync(0xffffffffu, (v >> b) & 1);
    off += __popc(m & lt) << b;
    total += __popc(m) << b;
  }
  return off;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

struct __align__(16) StagedTwig {
  float4 c;   // (coc - g) rounded from FP64 (k_walk_group64: its negation), charge
  float4 m0;  // px py pz 3qxx
  float4 m1;  // 3qyy 3qzz 1.5qxy 1.5qyz
  float4 m2;  // 1.5qzx, trace, charge, -
};
// the strict form's twig record: the FP64 node centre, then the moments
struct __align__(16) StagedTwigS {
  double cx, cy, cz;
  float pad[2];
  float4 m0, m1, m2;
};
struct __align__(16) StagedLeaf {
  float4 c;          // (x - g) rounded from FP64, charge
  double x, y, z;    // FP64 position, for the exact self test
  int box, pad;      // the record's box (walk_block.cu)
};

// The targets of one lane of a 64-target bucket: offsets from the group centre
// and (the strict form's) positions minus the box vector.
struct Targets64 {
  float rxa, rya, rza, rxb, ryb, rzb;
  double sxa, sya, sza, sxb, syb, szb;
};
template <bool kStrict>
using TwigRec64 = typename std::conditional<kStrict, StagedTwigS, StagedTwig>::type;

// Evaluates n staged twig records from ring position head on (two contiguous
// runs at most) for the lane's pair of targets, and adds the batch's sums to
// the FP64 sums acc[k * stride] (E and phi of the first target, then of the
// second).
template <bool kStrict>
__device__ __forceinline__ void twig_batch64(const TwigRec64<kStrict>* ring, int head, int n,
                                             int cap, const Targets64& T, float eps2,
                                             double* acc, int stride) {
  float2 PX = f2(0.f), PY = f2(0.f), PZ = f2(0.f), PP = f2(0.f);
  const float2 E2 = f2(eps2);
  const int n1 = min(n, cap - head);
  const TwigRec64<kStrict>* r = ring + head;
  if constexpr (kStrict) {
    float2 CX = f2(0.f), CY = f2(0.f), CZ = f2(0.f), CP = f2(0.f);
    auto one = [&](const TwigRec64<kStrict>& q) {
      // target minus node centre in FP64, rounded once
      const float2 dx = make_float2((float)(T.sxa - q.cx), (float)(T.sxb - q.cx));
      const float2 dy = make_float2((float)(T.sya - q.cy), (float)(T.syb - q.cy));
      const float2 dz = make_float2((float)(T.sza - q.cz), (float)(T.szb - q.cz));
      float2 tx, ty, tz, tp;
      twig32x2_terms(q.m0, q.m1, q.m2, dx, dy, dz, E2, tx, ty, tz, tp);
      kahan2(PX, CX, tx);
      kahan2(PY, CY, ty);
      kahan2(PZ, CZ, tz);
      kahan2(PP, CP, tp);
    };
#pragma unroll 4
    for (int j = 0; j < n1; ++j) one(r[j]);
#pragma unroll 2
    for (int j = 0; j < n - n1; ++j) one(ring[j]);
    // the compensated sum is s - c
    acc[0] += (double)PX.x - (double)CX.x;
    acc[stride] += (double)PY.x - (double)CY.x;
    acc[2 * stride] += (double)PZ.x - (double)CZ.x;
    acc[3 * stride] += (double)PP.x - (double)CP.x;
    acc[4 * stride] += (double)PX.y - (double)CX.y;
    acc[5 * stride] += (double)PY.y - (double)CY.y;
    acc[6 * stride] += (double)PZ.y - (double)CZ.y;
    acc[7 * stride] += (double)PP.y - (double)CP.y;
  } else {
    const float2 RX = make_float2(T.rxa, T.rxb), RY = make_float2(T.rya, T.ryb),
                 RZ = make_float2(T.rza, T.rzb);
    auto one = [&](const TwigRec64<kStrict>& q) {
      // c is the negated offset: one packed add per axis
      const float4 c = q.c, m0 = q.m0, m1 = q.m1, m2 = q.m2;
      twig32x2(m0, m1, m2, __fadd2_rn(RX, f2(c.x)), __fadd2_rn(RY, f2(c.y)),
               __fadd2_rn(RZ, f2(c.z)), E2, PX, PY, PZ, PP);
    };
#pragma unroll 16
    for (int j = 0; j < n1; ++j) one(r[j]);
#pragma unroll 4
    for (int j = 0; j < n - n1; ++j) one(ring[j]);
    acc[0] += (double)PX.x;
    acc[stride] += (double)PY.x;
    acc[2 * stride] += (double)PZ.x;
    acc[3 * stride] += (double)PP.x;
    acc[4 * stride] += (double)PX.y;
    acc[5 * stride] += (double)PY.y;
    acc[6 * stride] += (double)PZ.y;
    acc[7 * stride] += (double)PP.y;
  }
}

// The same for n <= 32 staged leaf records (v1: the lane has a second target;
// ta, tb: its targets; vb(record): the record's box vector).  Returns how many
// of the pairs are a target and its own leaf (no interaction).
template <bool kStrict, class F>
__device__ __forceinline__ unsigned leaf_batch64(const StagedLeaf* ring, int head, int n, int cap,
                                                 const Targets64& T, bool v1, const MixArgs& A,
                                                 int64_t ta, int64_t tb, F&& vb, double* acc,
                                                 int stride) {
  float2 PX = f2(0.f), PY = f2(0.f), PZ = f2(0.f), PP = f2(0.f);
  const float2 E2 = f2(A.eps2);
  const int n1 = min(n, cap - head);
  const StagedLeaf* r = ring + head;
  unsigned nuse = 0;
  if constexpr (kStrict) {
    float2 CX = f2(0.f), CY = f2(0.f), CZ = f2(0.f), CP = f2(0.f);
    auto leaf = [&](const StagedLeaf& r) {
      const double exa = T.sxa - r.x, eya = T.sya - r.y, eza = T.sza - r.z;
      const double exb = T.sxb - r.x, eyb = T.syb - r.y, ezb = T.szb - r.z;
      float2 wq = f2(r.c.w);
      // self: dist2 == 0 in FP64 (module_tree_walk_pthreads.f90:625)
      if (exa == 0.0 && eya == 0.0 && eza == 0.0) { wq.x = 0.f; ++nuse; }
      if (v1 && exb == 0.0 && eyb == 0.0 && ezb == 0.0) { wq.y = 0.f; ++nuse; }
      const float2 dx = make_float2((float)exa, (float)exb);
      const float2 dy = make_float2((float)eya, (float)eyb);
      const float2 dz = make_float2((float)eza, (float)ezb);
      const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, E2)));
      const float2 ri = make_float2(r2.x > 0.f ? rsqrt_ftz(r2.x) : 0.f, r2.y > 0.f ? rsqrt_ftz(r2.y) : 0.f);
      const float2 qr = __fmul2_rn(wq, ri);
      const float2 qr3 = __fmul2_rn(__fmul2_rn(qr, ri), ri);
      kahan2(PP, CP, qr);
      kahan2(PX, CX, __fmul2_rn(qr3, dx));
      kahan2(PY, CY, __fmul2_rn(qr3, dy));
      kahan2(PZ, CZ, __fmul2_rn(qr3, dz));
    };
#pragma unroll 4
    for (int j = 0; j < n1; ++j) leaf(r[j]);
#pragma unroll 2
    for (int j = 0; j < n - n1; ++j) leaf(ring[j]);
    acc[0] += (double)PX.x - (double)CX.x;
    acc[stride] += (double)PY.x - (double)CY.x;
    acc[2 * stride] += (double)PZ.x - (double)CZ.x;
    acc[3 * stride] += (double)PP.x - (double)CP.x;
    acc[4 * stride] += (double)PX.y - (double)CX.y;
    acc[5 * stride] += (double)PY.y - (double)CY.y;
    acc[6 * stride] += (double)PZ.y - (double)CZ.y;
    acc[7 * stride] += (double)PP.y - (double)CP.y;
  } else {
    const float2 RX = make_float2(T.rxa, T.rxb), RY = make_float2(T.rya, T.ryb),
                 RZ = make_float2(T.rza, T.rzb);
    auto leaf = [&](const StagedLeaf& r, int k, unsigned& pend) {
      const float4 c = r.c;
      const float2 dx = __fadd2_rn(RX, f2(-c.x)), dy = __fadd2_rn(RY, f2(-c.y)),
                   dz = __fadd2_rn(RZ, f2(-c.z));
      const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
      // a zero FP32 offset (the target's own leaf, or two points closer
      // than FP32 resolves at the group scale) enters with charge 0 here,
      // without a branch, and is decided and evaluated in FP64 after the
      // batch (pend: one bit per record of the batch)
      const bool za = d2.x == 0.f, zb = v1 && d2.y == 0.f;
      pend |= (za || zb) ? (1u << k) : 0u;
      const float2 wq = make_float2(za ? 0.f : c.w, zb ? 0.f : c.w);
      // the pair's leaf32 in packed FP32.  A zero r2 (eps2 = 0) comes with charge 0
      // and gives no contribution: the bound keeps its rsqrt finite, and lies below
      // any square of an offset that is not zero in FP32 at a scale >= 1e-18
      const float2 r2 = __fadd2_rn(d2, E2);
      const float2 ri = make_float2(rsqrt_ftz(fmaxf(r2.x, 1e-37f)), rsqrt_ftz(fmaxf(r2.y, 1e-37f)));
      const float2 qr = __fmul2_rn(wq, ri);
      const float2 qr3 = __fmul2_rn(__fmul2_rn(qr, ri), ri);
      PP = __fadd2_rn(PP, qr);
      PX = __ffma2_rn(qr3, dx, PX);
      PY = __ffma2_rn(qr3, dy, PY);
      PZ = __ffma2_rn(qr3, dz, PZ);
    };
    unsigned pend = 0;
#pragma unroll 4
    for (int j = 0; j < n1; ++j) leaf(r[j], j, pend);
#pragma unroll 2
    for (int j = 0; j < n - n1; ++j) leaf(ring[j], n1 + j, pend);
    // the zero-offset pairs: self when the FP64 offset is exactly zero
    // (dist2 == 0, module_tree_walk_pthreads.f90:625), else evaluated on
    // the FP64 offset rounded once
    while (pend) {
      const int k = __ffs(pend) - 1;
      pend &= pend - 1;
      const StagedLeaf& rr = ring[(head + k) & (cap - 1)];
      const float4 c = rr.c;
      const double3 v = vb(rr);
      for (int s2 = 0; s2 < 2; ++s2) {
        if (s2 == 1 && !v1) break;
        const float fx = (s2 ? T.rxb : T.rxa) - c.x, fy = (s2 ? T.ryb : T.rya) - c.y,
                    fz = (s2 ? T.rzb : T.rza) - c.z;
        if (fx * fx + fy * fy + fz * fz != 0.f) continue;  // evaluated in the batch
        const int64_t tt = s2 ? tb : ta;
        const double ex = (A.tx[tt] - v.x) - rr.x, ey = (A.ty[tt] - v.y) - rr.y,
                     ez = (A.tz[tt] - v.z) - rr.z;
        if (ex == 0.0 && ey == 0.0 && ez == 0.0) {
          ++nuse;
          continue;
        }
        float ax = 0.f, ay = 0.f, az = 0.f, ap = 0.f;
        leaf32(c.w, (float)ex, (float)ey, (float)ez, A.eps2, ax, ay, az, ap);
        if (s2) { PX.y += ax; PY.y += ay; PZ.y += az; PP.y += ap; }
        else { PX.x += ax; PY.x += ay; PZ.x += az; PP.x += ap; }
      }
    }
    acc[0] += (double)PX.x;
    acc[stride] += (double)PY.x;
    acc[2 * stride] += (double)PZ.x;
    acc[3 * stride] += (double)PP.x;
    acc[4 * stride] += (double)PX.y;
    acc[5 * stride] += (double)PY.y;
    acc[6 * stride] += (double)PZ.y;
    acc[7 * stride] += (double)PP.y;
  }
  return nuse;
}

struct AdjMixArgs {
  int64_t nt;
  const double *tx, *ty, *tz;
  const double *gex, *gey, *gez, *gphi;
  const double4* nc4;
  const int2* meta;
  const float4* mom32;
  const int32_t* nleaves;
  const LevelRecord* drec;  // level-ordered node records with walk links (grow.cu)
  const double* bl2;
  const double* macb;
  const double* vbox;
  int nbox;
  float theta2, eps2;
  int64_t npart;
  double* adj;  // 16 doubles per node, level order: q, p(3), Q(6: xx yy zz xy yz zx), coc(3), abs_charge, pad
  unsigned long long* counters;
  uint32_t* status;
  unsigned int* queue;
};

constexpr int kNAdj = 16;

struct __align__(16) StagedLeafA {
  float4 c;        // (x - g) rounded from FP64, charge
  double x, y, z;  // FP64 position, for the exact self test
  int node;
  int pad;
};

__device__ __forceinline__ void adj_add(double* __restrict__ a, float2 v) {
  const double s = (double)v.x + (double)v.y;
  if (s != 0.0) atomicAdd(a, s);
}

// one staged twig record's adjoint, summed over the bucket's 64 targets (tg:
// the pre-paired offsets and gradients) and added to the node's FP64 record
template <bool kWithE>
__device__ __forceinline__ void adj_twig_record(const StagedTwig& r,
                                                const float4 (*tg)[kWithE ? 4 : 2], float2 E2,
                                                double* __restrict__ adj) {
  const float4 c = r.c, m0 = r.m0, m1 = r.m1, m2 = r.m2;
  const int node = __float_as_int(c.w);
  const float2 CX = f2(c.x), CY = f2(c.y), CZ = f2(c.z);  // d = r_t + c
  const float2 PX = f2(m0.x), PY = f2(m0.y), PZ = f2(m0.z);
  // -(p.d + tr) = (-p).d + (-tr): the negated dipole and trace, once per record
  const float2 NPX = f2(-m0.x), NPY = f2(-m0.y), NPZ = f2(-m0.z), NTR = f2(-m2.y);
  const float2 Txx = f2(m0.w), Tyy = f2(m1.x), Tzz = f2(m1.y), Txy = f2(m1.z),
               Tyz = f2(m1.w), Tzx = f2(m2.x), Q = f2(m2.z);
  float2 aq = f2(0.f), apx = f2(0.f), apy = f2(0.f), apz = f2(0.f), aS = f2(0.f);
  float2 axx = f2(0.f), ayy = f2(0.f), azz = f2(0.f), axy = f2(0.f), ayz = f2(0.f),
         azx = f2(0.f), acx = f2(0.f), acy = f2(0.f), acz = f2(0.f);
  float2 aGx = f2(0.f), aGy = f2(0.f), aGz = f2(0.f);  // sum of 2 R2 g (with E)
#pragma unroll 4
  for (int p = 0; p < 32; ++p) {
    const float4 ta4 = tg[p][0], tb4 = tg[p][1];
    const float2 dx = __fadd2_rn(make_float2(ta4.x, ta4.y), CX);
    const float2 dy = __fadd2_rn(make_float2(ta4.z, ta4.w), CY);
    const float2 dz = __fadd2_rn(make_float2(tb4.x, tb4.y), CZ);
    const float2 gp = make_float2(tb4.z, tb4.w);
    const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, E2)));
    const float2 R0 = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
    const float2 i2 = __fmul2_rn(R0, R0);
    const float2 R1 = __fmul2_rn(R0, i2);
    // scaled radial factors: T3 = 3 R2, F5 = 5 R3
    const float2 T3 = __fmul2_rn(R1, __fmul2_rn(f2(3.f), i2));
    const float2 F5 = __fmul2_rn(T3, __fmul2_rn(f2(5.f / 3.f), i2));
    const float2 vx = __ffma2_rn(Txx, dx, __ffma2_rn(Txy, dy, __fmul2_rn(Tzx, dz)));
    const float2 vy = __ffma2_rn(Txy, dx, __ffma2_rn(Tyy, dy, __fmul2_rn(Tyz, dz)));
    const float2 vz = __ffma2_rn(Tzx, dx, __ffma2_rn(Tyz, dy, __fmul2_rn(Tzz, dz)));
    const float2 dTd = __ffma2_rn(dx, vx, __ffma2_rn(dy, vy, __fmul2_rn(dz, vz)));
    const float2 nu = __ffma2_rn(NPX, dx, __ffma2_rn(NPY, dy, __ffma2_rn(NPZ, dz, NTR)));
    // ce = q R1 - 3 R2 (p.d + tr) + 5 R3 dTd
    const float2 ce = __ffma2_rn(Q, R1, __ffma2_rn(T3, nu, __fmul2_rn(F5, dTd)));
    const float2 s1 = __fmul2_rn(gp, R1);
    float2 s3 = __fmul2_rn(gp, T3);
    aq = __ffma2_rn(gp, R0, aq);
    aS = __fadd2_rn(aS, s1);
    float2 kd = __fmul2_rn(gp, ce);                        // coefficient of d in cocbar
    float2 kv = __fmul2_rn(f2(-2.f / 3.f), s3);            // of v
    float2 ex_ = f2(0.f), ey_ = f2(0.f), ez_ = f2(0.f);     // -3 R2 g
    float2 ppx = s1;                                        // coefficient of -d in pbar
    if constexpr (kWithE) {
      const float4 tc4 = tg[p][2], td4 = tg[p][3];
      const float2 gxx = make_float2(tc4.x, tc4.y), gyy = make_float2(tc4.z, tc4.w),
                   gzz = make_float2(td4.x, td4.y);
      const float2 ga = __ffma2_rn(gxx, dx, __ffma2_rn(gyy, dy, __fmul2_rn(gzz, dz)));
      const float2 F15 = __fmul2_rn(f2(3.f), F5);
      const float2 F10n = __fmul2_rn(f2(-2.f), F5);
      const float2 S35 = __fmul2_rn(F5, __fmul2_rn(f2(7.f), i2));  // 35 R4
      aq = __ffma2_rn(ga, R1, aq);
      // pbar += R1 g - 3 ga R2 d, kept as -pbar
      const float2 h = __fmul2_rn(ga, T3);  // 3 ga R2
      const float2 nR1 = __fmul2_rn(f2(-1.f), R1);
      apx = __ffma2_rn(nR1, gxx, apx);
      apy = __ffma2_rn(nR1, gyy, apy);
      apz = __ffma2_rn(nR1, gzz, apz);
      ppx = __fadd2_rn(s1, h);
      // Qbar: 15 ga R3 d d - 3 R2 (g d + d g + ga I)
      s3 = __ffma2_rn(F15, ga, s3);
      const float2 nT3 = __fmul2_rn(f2(-1.f), T3);
      ex_ = __fmul2_rn(nT3, gxx);
      ey_ = __fmul2_rn(nT3, gyy);
      ez_ = __fmul2_rn(nT3, gzz);
      aS = __fadd2_rn(aS, h);  // the delta_kl and the p terms share 3 ga R2
      // cocbar: cd d + cg g + 3 R2 ga p - 10 R3 ga v + 2 R2 T g, cg = -ce,
      // cd = ga (3 q R2 - 15 R3 u + 35 R4 dTd) + 3 R2 (g.p) - 10 R3 (g.v);
      // T g is node-constant: the batch sums 2 R2 g (aG) and applies T once
      const float2 gP = __ffma2_rn(gxx, PX, __ffma2_rn(gyy, PY, __fmul2_rn(gzz, PZ)));
      const float2 gv = __ffma2_rn(gxx, vx, __ffma2_rn(gyy, vy, __fmul2_rn(gzz, vz)));
      const float2 inner = __ffma2_rn(Q, T3, __ffma2_rn(F15, nu, __fmul2_rn(S35, dTd)));
      const float2 cd = __ffma2_rn(ga, inner, __ffma2_rn(T3, gP, __fmul2_rn(F10n, gv)));
      kd = __fadd2_rn(kd, cd);
      kv = __ffma2_rn(F10n, ga, kv);
      const float2 R2x2 = __fmul2_rn(f2(2.f / 3.f), T3);
      aGx = __ffma2_rn(R2x2, gxx, aGx);
      aGy = __ffma2_rn(R2x2, gyy, aGy);
      aGz = __ffma2_rn(R2x2, gzz, aGz);
      const float2 nce = __fmul2_rn(f2(-1.f), ce);
      acx = __ffma2_rn(nce, gxx, acx);
      acy = __ffma2_rn(nce, gyy, acy);
      acz = __ffma2_rn(nce, gzz, acz);
    }
    apx = __ffma2_rn(ppx, dx, apx);
    apy = __ffma2_rn(ppx, dy, apy);
    apz = __ffma2_rn(ppx, dz, apz);
    // Qbar's d d terms and (with E) the g d terms:
    //   kl += (s3 d_k + e_k) d_l + e_l d_k,  e = -3 R2 g
    const float2 wx = __ffma2_rn(s3, dx, ex_), wy = __ffma2_rn(s3, dy, ey_),
                 wz = __ffma2_rn(s3, dz, ez_);
    axx = __ffma2_rn(__fadd2_rn(wx, ex_), dx, axx);
    ayy = __ffma2_rn(__fadd2_rn(wy, ey_), dy, ayy);
    azz = __ffma2_rn(__fadd2_rn(wz, ez_), dz, azz);
    axy = __ffma2_rn(wx, dy, __ffma2_rn(ey_, dx, axy));
    ayz = __ffma2_rn(wy, dz, __ffma2_rn(ez_, dy, ayz));
    azx = __ffma2_rn(wz, dx, __ffma2_rn(ex_, dz, azx));
    acx = __ffma2_rn(kd, dx, __ffma2_rn(kv, vx, acx));
    acy = __ffma2_rn(kd, dy, __ffma2_rn(kv, vy, acy));
    acz = __ffma2_rn(kd, dz, __ffma2_rn(kv, vz, acz));
  }
  double* a = adj + (int64_t)kNAdj * node;
  // the node-constant factors: the delta_kl terms and R1 p (with E also 3 R2 ga p)
  const double S = (double)aS.x + (double)aS.y;
  adj_add(a + 0, aq);
  adj_add(a + 1, make_float2(-apx.x, -apx.y));
  adj_add(a + 2, make_float2(-apy.x, -apy.y));
  adj_add(a + 3, make_float2(-apz.x, -apz.y));
  if (S != 0.0) {
    atomicAdd(a + 4, (double)axx.x + (double)axx.y - S);
    atomicAdd(a + 5, (double)ayy.x + (double)ayy.y - S);
    atomicAdd(a + 6, (double)azz.x + (double)azz.y - S);
  } else {
    adj_add(a + 4, axx);
    adj_add(a + 5, ayy);
    adj_add(a + 6, azz);
  }
  adj_add(a + 7, axy);
  adj_add(a + 8, ayz);
  adj_add(a + 9, azx);
  double cx = (double)acx.x + (double)acx.y + S * (double)m0.x;
  double cy = (double)acy.x + (double)acy.y + S * (double)m0.y;
  double cz = (double)acz.x + (double)acz.y + S * (double)m0.z;
  if constexpr (kWithE) {
    // + T (sum of 2 R2 g)
    const double Gx = (double)aGx.x + (double)aGx.y, Gy = (double)aGy.x + (double)aGy.y,
                 Gz = (double)aGz.x + (double)aGz.y;
    cx += (double)m0.w * Gx + (double)m1.z * Gy + (double)m2.x * Gz;
    cy += (double)m1.z * Gx + (double)m1.x * Gy + (double)m1.w * Gz;
    cz += (double)m2.x * Gx + (double)m1.w * Gy + (double)m1.y * Gz;
  }
  if (cx != 0.0) atomicAdd(a + 10, cx);
  if (cy != 0.0) atomicAdd(a + 11, cy);
  if (cz != 0.0) atomicAdd(a + 12, cz);
}

// one staged leaf record's adjoint; v: the record's box vector, t0: the
// bucket's first target
template <bool kWithE>
__device__ __forceinline__ void adj_leaf_record(const StagedLeafA& r,
                                                const float4 (*tg)[kWithE ? 4 : 2], float2 E2,
                                                const AdjMixArgs& A, int64_t t0, double3 v) {
  const float4 c = r.c;
  const float2 NCX = f2(-c.x), NCY = f2(-c.y), NCZ = f2(-c.z);  // d = r_t - c
  float2 aq = f2(0.f), acx = f2(0.f), acy = f2(0.f), acz = f2(0.f);
  unsigned long long pend = 0ull;  // targets at a zero FP32 offset (bit 2p + half)
#pragma unroll 2
  for (int p = 0; p < 32; ++p) {
    const float4 ta4 = tg[p][0], tb4 = tg[p][1];
    const float2 dx = __fadd2_rn(make_float2(ta4.x, ta4.y), NCX);
    const float2 dy = __fadd2_rn(make_float2(ta4.z, ta4.w), NCY);
    const float2 dz = __fadd2_rn(make_float2(tb4.x, tb4.y), NCZ);
    const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
    const bool za = d2.x == 0.f, zb = d2.y == 0.f;
    pend |= (za ? 1ull << (2 * p) : 0ull) | (zb ? 2ull << (2 * p) : 0ull);
    const float2 gp = make_float2(za ? 0.f : tb4.z, zb ? 0.f : tb4.w);
    const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, E2)));
    const float2 R0 = make_float2(r2.x > 0.f ? rsqrt_ftz(r2.x) : 0.f,
                                  r2.y > 0.f ? rsqrt_ftz(r2.y) : 0.f);
    const float2 R1 = __fmul2_rn(R0, __fmul2_rn(R0, R0));
    aq = __ffma2_rn(gp, R0, aq);
    float2 k = __fmul2_rn(gp, R1);
    if constexpr (kWithE) {
      const float4 tc4 = tg[p][2], td4 = tg[p][3];
      const float2 gxx = make_float2(za ? 0.f : tc4.x, zb ? 0.f : tc4.y);
      const float2 gyy = make_float2(za ? 0.f : tc4.z, zb ? 0.f : tc4.w);
      const float2 gzz = make_float2(za ? 0.f : td4.x, zb ? 0.f : td4.y);
      const float2 ga = __ffma2_rn(gxx, dx, __ffma2_rn(gyy, dy, __fmul2_rn(gzz, dz)));
      const float2 R2 = __fmul2_rn(R1, __fmul2_rn(R0, R0));
      aq = __ffma2_rn(ga, R1, aq);
      k = __ffma2_rn(__fmul2_rn(f2(3.f), ga), R2, k);
      const float2 nR1 = __fmul2_rn(f2(-1.f), R1);
      acx = __ffma2_rn(nR1, gxx, acx);
      acy = __ffma2_rn(nR1, gyy, acy);
      acz = __ffma2_rn(nR1, gzz, acz);
    }
    acx = __ffma2_rn(k, dx, acx);
    acy = __ffma2_rn(k, dy, acy);
    acz = __ffma2_rn(k, dz, acz);
  }
  // zero FP32 offsets: the target's own leaf (no interaction, FP64
  // dist2 == 0) or a point closer than FP32 resolves at the group
  // scale, evaluated on the FP64 offset rounded once
  float sq = 0.f, scx = 0.f, scy = 0.f, scz = 0.f;
  while (pend) {
    const int bit = __ffsll((long long)pend) - 1;
    pend &= pend - 1;
    const int64_t t = t0 + (bit >> 1) + 32 * (bit & 1);
    const double ex = (A.tx[t] - v.x) - r.x, ey = (A.ty[t] - v.y) - r.y,
                 ez = (A.tz[t] - v.z) - r.z;
    if (ex == 0.0 && ey == 0.0 && ez == 0.0) continue;
    const float dx = (float)ex, dy = (float)ey, dz = (float)ez;
    const float gp = (float)A.gphi[t];
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, A.eps2)));
    const float R0 = rsqrt_ftz(r2), R1 = R0 * R0 * R0;
    sq = fmaf(gp, R0, sq);
    float k = gp * R1;
    if constexpr (kWithE) {
      const float gx = (float)A.gex[t], gy = (float)A.gey[t], gz = (float)A.gez[t];
      const float ga = fmaf(gx, dx, fmaf(gy, dy, gz * dz));
      sq = fmaf(ga, R1, sq);
      k = fmaf(3.f * ga, R1 * R0 * R0, k);
      scx = fmaf(-R1, gx, scx);
      scy = fmaf(-R1, gy, scy);
      scz = fmaf(-R1, gz, scz);
    }
    scx = fmaf(k, dx, scx);
    scy = fmaf(k, dy, scy);
    scz = fmaf(k, dz, scz);
  }
  double* a = A.adj + (int64_t)kNAdj * r.node;
  const double q = (double)c.w;
  const double vq = (double)aq.x + (double)aq.y + (double)sq;
  if (vq != 0.0) atomicAdd(a + 0, vq);
  const double cx = q * ((double)acx.x + (double)acx.y + (double)scx);
  const double cy = q * ((double)acy.x + (double)acy.y + (double)scy);
  const double cz = q * ((double)acz.x + (double)acz.y + (double)scz);
  if (cx != 0.0) atomicAdd(a + 10, cx);
  if (cy != 0.0) atomicAdd(a + 11, cy);
  if (cz != 0.0) atomicAdd(a + 12, cz);
}

// ---- walk_block.cu: one block (or cluster) per bucket, for few buckets ----
struct BlockShape {
  int warps = 0;  // per block
  int parts = 1;  // blocks of the cluster that shares a bucket
};
// Whether nt targets on a tree of npart particles are walked by blocks, and how.
// A bucket's sums depend on the shape only (FP32 batches), so calls that must
// give the same fields pass the same nt here.
enum class BlockWalk { kDefault, kStrict, kAdjoint };
bool block_walk_shape(int64_t nt, int64_t npart, BlockWalk kind, bool keyed, BlockShape* sh);
bool launch_walk_block64(Ctx* c, const MixArgs& A, const BlockShape& sh, bool strict, int* stack,
                         cudaStream_t s);
bool launch_adj_block64(Ctx* c, const AdjMixArgs& A, const BlockShape& sh, bool with_e, int* stack,
                        cudaStream_t s);

}  // namespace pepcg
