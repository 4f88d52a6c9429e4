// Force walk of the B200 Barnes-Hut path.
//
// What a target receives is exactly the reference's interaction list
// (GroupWalker, grouped_ttg.h:204-289): the bounding box of the target's
// particles (BBox, multipole.h:115-142) is tested against the visited nodes
// with mac_accept_bbox (multipole.h:151-153, strict theta^2 near^2 > edge^2,
// in FP64); leaves are tested too; accepted nodes are cell interactions
// (quadrupole, accel_from_source multipole.h:171-200, or monopoles in
// no-quad mode); everything else is opened - interior nodes push their
// children, leaves contribute their particles directly, the target's own
// leaf included (its self term is 0 with softening and masked at r^2 = 0
// without, accumulate_list grouped_ttg.h:117-163).
//
// One warp per walk GROUP (a run of consecutive targets of one system, at
// most kGroupMax particles and kMaxTargets targets, k_pack_groups), sharing
// the walk among the group's targets as GroupWalker::visit does, taken to
// every level: one traversal from the root whose stack entries carry the
// mask of targets that still need the nodes.  A node accepted for the
// group's bounding box is accepted by every target in the mask; one rejected
// for every point of it (mac_reject_all, multipole.h:158-160) is opened by
// all of them; otherwise each target tests its own box.  Sources every
// target of the group takes go to the warp's dense list, sources only some
// take to its partial list as (node or leaf run, target mask).  Each target's
// list is the same as a separate walk of its box from the root would build.
//
// Then the lists are evaluated: the dense one once against all the group's
// particles, the partial one once per target, which takes its own entries.
// A list pass gathers the picked sources into batches (64 cells or 128
// particles in split precision, 32 or 64 in FP64).  Traversal and evaluation
// take turns, so that neither holds registers or shared memory of the other.
//
// Split precision: sources and targets become FP32 offsets from the
// particles' bounding-box centre (the subtraction in FP64), staged once per
// batch in shared memory; interactions are packed FP32 FMA +
// rsqrt.approx.ftz, lanes laid out as (target, source subset) (SplitEval
// below); FP32 partials go into FP64 sums every 32 or more terms.  The
// kick/drift of integrate_ttg.h:74-77 is applied in FP64 in the epilogue.
#include "bhg_walk.cuh"
#include "bhg_lists.h"

#include <algorithm>
#include <type_traits>

namespace bhg {

constexpr int kStackCap = 176;       // per-warp traversal stack: runs of sibling nodes
constexpr int kRing = 160;           // sources picked for the next batch (a batch of up to 128, less one, + 32)
constexpr int kStageBytes = 2560;    // staged sources of one batch
// Lists are two-ended arrays of uint2: cells from the front, runs of particles
// (opened leaves) from the back.  The dense list (sources every target of
// the group takes): (node, 1) and (first particle, count).  The partial list
// (sources some targets take): (node, target mask) and (first particle, mask
// | count << kCountShift), or (leaf node, mask | kByNode << kCountShift) for
// a leaf of kByNode particles or more.
constexpr int kCountShift = 24;
constexpr uint32_t kMaskBits = (1u << kCountShift) - 1u;
constexpr uint32_t kByNode = 255;
static_assert(kMaxTargets <= kCountShift, "target masks and counts share a word");
constexpr uint32_t kDenseCap = 2048;  // entries of a dense list (16 KB)
// a group's list lengths are cells | runs << 16 (two-pass schedule)
static_assert(kListCap < 0xfefe, "list lengths never look pending, nor lost");
// a traversal step pops at most (free entries - kLevels - 1) nodes, one at
// least, and every popped node pushes at most one run of children, so that
// one-node steps (depth first, at most one run per level) never overflow
static_assert(kStackCap >= 32 + 2 * (kLevels + 1), "the stack holds a step's pushes");

struct Walk {
  uint32_t top, steps;          // stack entries; steps so far
  uint32_t ndc, ndr, npc, npr;  // dense cells and runs, partial cells and runs
};

// Jobs of the walk (k_walk): a group's traversal (and whatever passes no
// other job takes), a group's dense pass beside it, a target's pass.
enum : uint32_t { kWholeJob, kDenseJob, kTargetJob };
// A group's progress (kListPending before the walk): cells in its dense list so far; or kFinal | runs << 12 | cells; or
// kAborted, when the traversal paused and evaluates its lists itself.
constexpr uint32_t kFinal = 1u << 31, kAborted = 1u << 30;
static_assert(kDenseCap < 1u << 12, "two lengths and the flags share a word");

// A warp's job, kept in shared memory (every lane writes the same values, a
// __syncwarp away from reads of older ones): the evaluation loops need the
// registers.
struct Job {
  uint32_t gi, ti;         // walk group; target (target jobs)
  uint32_t t0, k, p0, sys;  // the group's first target, targets, first particle, system
  uint32_t n, b0;          // particles; a large target's batch start
  uint32_t pass1;          // the last pass to run
  uint32_t more, kind;     // the traversal paused; kWholeJob, kDenseJob or kTargetJob
  uint32_t poll, aborted;  // dense jobs: cells are still to come; the traversal paused
  uint32_t left, told;     // left to the dense job; the traversal's cells published so far
  uint2 *dense, *partial;  // the lists
  Walk w;
};

struct WarpSmem {
  uint2 stack[kStackCap];  // run of sibling nodes: (first node, targets that still need them | nodes << 24)
  alignas(16) unsigned char stage[kStageBytes];  // a batch's staged sources; scratch of a traversal step
  double sums[6][32];        // FP64 sums of the lanes (evaluators)
  double acc[kGroupMax][3];  // FP64 sum per particle of the group
  double tlo[kMaxTargets][3], thi[kMaxTargets][3];  // the targets' particle boxes
  double glo[3], ghi[3];                            // the group's particle box
  double centre[3], scale, scale2, eps2;            // evaluators' reference point and units
  unsigned long long ncell, npart;                  // interactions of this warp
  unsigned long long kept[2];                       // of them, before a dense job that may be aborted
  Job job;
  uint32_t tbeg[kMaxTargets], tcnt[kMaxTargets];    // the targets' particles
  uint32_t ring[kRing];
  uint32_t delta[32];  // runs of a window: first particle less the particles of the runs before it
};
constexpr size_t kWalkSmem = sizeof(WarpSmem) * kWalkWarps;
// six blocks per SM: 228 KB, of which each block takes 1 KB for the system
static_assert(6 * (kWalkSmem + 1024) <= 228 * 1024, "shared memory of 24 warps per SM");

// Scratch of a traversal step (in WarpSmem::stage): the nodes that targets
// test on their own, and the targets that accept them.
struct StepScratch {
  float4 node[32];   // centre of mass, near^2 above which it is accepted
  float reject[32];  // near^2 below which it is not
  uint32_t id[32];
  uint32_t accepts[32];
};
static_assert(sizeof(StepScratch) <= kStageBytes && kGroupMax * 3 * 8 <= kStageBytes, "scratch in the staging area");

// ---------------------------------------------------------------------------
// Evaluators of the lists' sources.

// Two FP32 values in one 64-bit register: the SM's packed FP32 instructions
// (add, mul, fma .f32x2) work on both halves in one issue slot, each half
// rounded as the scalar instruction rounds it.
using f2 = unsigned long long;
__device__ __forceinline__ f2 f2_pack(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(f2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Split precision.  Sources are staged once per batch in shared memory as
// FP32 values relative to the walk box's centre (the subtraction in FP64),
// two sources to a record of packed pairs, and the warp is laid out as a grid
// of lanes: each lane owns two targets and one of ng lane groups, which split
// the batch's records between them (group g takes records g, g + ng, ...).
// Every lane reads the records it needs from shared memory (all lanes of a
// group read the same record: a broadcast), so a source costs one global
// gather per warp, not one per lane group, and the lanes never exchange
// partial sums inside a batch.  A loop iteration evaluates the four
// interactions of a record's two sources with the lane's two targets in
// packed FP32 arithmetic.  The FP32 partials (per target one for the first
// and one for the second source of the records) are added into per-lane FP64
// sums, each on its own, once they hold 32 or more terms (95 at most: 31 held
// over and a full batch of particles in one lane group) and at the end of the
// list; then the lane groups' FP64 sums are added in group order
// (deterministic) into the targets' FP64 sums.
// What bounds it: issue slots and latency, so halving the FP32 instructions
// pays although the FMA pipe's own rate stays the same.  Walk per evaluation,
// scalar / packed, with 16 warps per SM: 32.9 / 30.5 ms at 4M (leaf 16), 6.53
// / 5.52 at 1M with leaf 48, 4.04 / 3.35 at 1M with monopoles; warp
// instructions of a 1M walk 5.48e9 / 4.16e9.
// The units of FP32 arithmetic on offsets in a system of half width hw: a
// power of two near its size (see SplitEval).
__device__ __forceinline__ void set_units(WarpSmem& S, double hw) {
  int k = hw > 0.0 ? ilogb(hw) : 0;
  k = k < -100 ? -100 : (k > 100 ? 100 : k);
  S.scale = ldexp(1.0, -k);       // offsets d' = d * scale
  S.scale2 = ldexp(1.0, -2 * k);  // a = a' * scale^2 (a' = m d' / r'^3 = a / scale^2), Q' = Q * scale^2
}

// The lane groups' sums (S.sums; lane g * lpg + l: targets l and l + lpg),
// added in group order into the targets' FP64 sums out[0 .. tb).
__device__ __forceinline__ void add_group_sums(const WarpSmem& S, int lane, int tb, int lpg, int ng, double (*out)[3]) {
  for (int t = lane; t < tb; t += 32) {
    const int k = t >= lpg ? 3 : 0, sl = k ? t - lpg : t;
    double x = 0.0, y = 0.0, z = 0.0;
    for (int g = 0; g < ng; ++g) {
      const int l = g * lpg + sl;
      x += S.sums[k][l], y += S.sums[k + 1][l], z += S.sums[k + 2][l];
    }
    out[t][0] += x, out[t][1] += y, out[t][2] += z;
  }
  __syncwarp();
}

template <bool QUAD>
struct SplitEval {
  static constexpr int kCellBatch = 64, kPartBatch = 128;
  static constexpr int kBlocksPerSm = 6;
  // FP32 partials go into the FP64 sums once a lane has added kFlushTerms
  // or more terms to them, and at the end of a list
  static constexpr int kFlushTerms = 32;
  // Staged records, one plane of 16 bytes per record for each two components:
  // cells (x, y) (z, m) (q0, q1) (q2, q3) (q4, q5), particles (x, y) (z, m).
  // A 16-byte stride keeps the lane groups' reads free of bank conflicts.
  static constexpr int kCellPlane = kCellBatch / 2, kPartPlane = kPartBatch / 2;
  static_assert(5 * 16 * kCellPlane <= kStageBytes && 2 * 16 * kPartPlane <= kStageBytes && kPartBatch + 31 < kRing,
                "batches too large");
  const WalkArgs& a;
  WarpSmem& S;
  // the FP32 arithmetic runs on offsets times a power of two near the
  // system's size (1 / 2^ilogb(domain half width)), so that r^-7 of the
  // smallest and largest systems stays inside FP32's range; the powers of two
  // make the scaling exact (rsqrt of an even power of two too), and the FP64
  // sums are scaled back.  The scales and the reference point (the box's
  // centre) stay in shared memory: no registers while a batch is evaluated.
  int lane, ng, inv_ng, first;
  f2 t0x, t0y, t0z, t1x, t1y, t1z;  // minus the targets' positions, in both halves (t1 = t0 where there is none)
  f2 a0x, a0y, a0z, a1x, a1y, a1z;  // FP32 partials
  int pend;  // terms in this lane's FP32 partials since the last flush (an upper bound, warp-uniform)

  // softening eps2_, after set_units
  __device__ SplitEval(const WalkArgs& args, WarpSmem& S_, int lane_, double eps2_)
      : a(args), S(S_), lane(lane_) {
    const double scale = S.scale;
    S.eps2 = eps2_ * (scale * scale);  // eps2' = eps2 * scale^2
  }

  // targets: particles p0 .. p0 + n - 1 (n <= 64), offsets from (x, y, z)
  __device__ void setup(uint32_t p0, int n, double x, double y, double z) {
    S.centre[0] = x, S.centre[1] = y, S.centre[2] = z;
    const int lpg = (n + 1) >> 1, inv = 65536 / lpg + 1;  // x / lpg = x * inv >> 16 for x <= 95
    const int g = lane * inv >> 16, t0 = lane - g * lpg, t1 = t0 + lpg < n ? t0 + lpg : t0;
    ng = 32 * inv >> 16;
    inv_ng = 65536 / ng + 1;
    first = g < ng ? g : 1 << 30;  // inactive lanes take no sources
    const double4 q0 = a.pm[p0 + t0], q1 = a.pm[p0 + t1];
    const double scale = S.scale;
    t0x = twice(__dsub_rn(x, q0.x) * scale), t0y = twice(__dsub_rn(y, q0.y) * scale);
    t0z = twice(__dsub_rn(z, q0.z) * scale);
    t1x = twice(__dsub_rn(x, q1.x) * scale), t1y = twice(__dsub_rn(y, q1.y) * scale);
    t1z = twice(__dsub_rn(z, q1.z) * scale);
    a0x = a0y = a0z = a1x = a1y = a1z = 0ull;
#pragma unroll
    for (int c = 0; c < 6; ++c) S.sums[c][lane] = 0.0;
    pend = 0;
  }

  static __device__ __forceinline__ f2 twice(double d) {
    const float f = (float)d;
    return f2_pack(f, f);
  }

  // one FP32 partial into its FP64 sum, each half widened on its own (added in
  // FP32 first, two halves of 32 terms would round like a chain of 64; 4M
  // 21.50 / 21.54 ms, 1M with monopoles 2.58 / 2.59)
  __device__ __forceinline__ void flush_one(f2& p, int c) const {
    float lo, hi;
    f2_unpack(p, lo, hi);
    S.sums[c][lane] += ((double)lo + (double)hi) * S.scale2;
    p = 0ull;
  }

  __device__ __forceinline__ void flush() {
    flush_one(a0x, 0), flush_one(a0y, 1), flush_one(a0z, 2);
    flush_one(a1x, 3), flush_one(a1y, 4), flush_one(a1z, 5);
    pend = 0;
  }

  // 1 / sqrt(r^2) of both halves (softened: r^2 > 0)
  static __device__ __forceinline__ f2 rsqrt2(f2 r2) {
    float lo, hi;
    f2_unpack(r2, lo, hi);
    return f2_pack(rsqrt_ftz(lo), rsqrt_ftz(hi));
  }

  // a record of two cells acting on the target at -(tx, ty, tz); the staged
  // quadrupoles are negated: n.. = -Q..
  __device__ __forceinline__ void cell_body(ulonglong2 xy, ulonglong2 zm, ulonglong2 n01, ulonglong2 n23,
                                            ulonglong2 n45, f2 e2, f2 tx, f2 ty, f2 tz, f2& ax, f2& ay, f2& az) const {
    const f2 dx = f2_add(xy.x, tx), dy = f2_add(xy.y, ty), dz = f2_add(zm.x, tz);
    const f2 r2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_fma(dz, dz, e2)));
    const f2 ri = rsqrt2(r2);
    const f2 ri2 = f2_mul(ri, ri);
    const f2 ri3 = f2_mul(ri, ri2);
    if (QUAD) {
      // Q = [[q0 q3 q4] [q3 q1 q5] [q4 q5 q2]]
      const f2 qx = f2_fma(n01.x, dx, f2_fma(n23.y, dy, f2_mul(n45.x, dz)));
      const f2 qy = f2_fma(n23.y, dx, f2_fma(n01.y, dy, f2_mul(n45.y, dz)));
      const f2 qz = f2_fma(n45.x, dx, f2_fma(n45.y, dy, f2_mul(n23.x, dz)));
      const f2 dqd = f2_fma(dx, qx, f2_fma(dy, qy, f2_mul(dz, qz)));
      const f2 ri5 = f2_mul(ri3, ri2);
      // m d / r^3 - Q d / r^5 + 2.5 (d Q d) d / r^7
      const f2 c = f2_fma(f2_mul(f2_pack(-2.5f, -2.5f), dqd), f2_mul(ri5, ri2), f2_mul(zm.y, ri3));
      ax = f2_fma(ri5, qx, f2_fma(c, dx, ax));
      ay = f2_fma(ri5, qy, f2_fma(c, dy, ay));
      az = f2_fma(ri5, qz, f2_fma(c, dz, az));
    } else {
      const f2 c = f2_mul(zm.y, ri3);
      ax = f2_fma(c, dx, ax), ay = f2_fma(c, dy, ay), az = f2_fma(c, dz, az);
    }
  }

  __device__ __forceinline__ void part_body(ulonglong2 xy, ulonglong2 zm, f2 e2, f2 tx, f2 ty, f2 tz, f2& ax, f2& ay,
                                            f2& az) const {
    const f2 dx = f2_add(xy.x, tx), dy = f2_add(xy.y, ty), dz = f2_add(zm.x, tz);
    const f2 r2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_fma(dz, dz, e2)));
    const f2 ri = rsqrt2(r2);
    const f2 c = f2_mul(f2_mul(zm.y, f2_mul(ri, ri)), ri);
    ax = f2_fma(c, dx, ax), ay = f2_fma(c, dy, ay), az = f2_fma(c, dz, az);
  }

  // one coordinate of two sources, as a packed pair of offsets
  __device__ __forceinline__ f2 offsets(double s0, double s1, double c, double scale) const {
    return f2_pack((float)(__dsub_rn(s0, c) * scale), (float)(__dsub_rn(s1, c) * scale));
  }

  // cells: node ids ring[0 .. cnt), cnt <= kCellBatch.  Lane r stages record
  // r: sources r and r + nrec (for the last record of an odd batch, one that
  // contributes exactly 0).
  __device__ __forceinline__ void cells(const uint32_t* ring, int cnt) {
    ulonglong2* rec = reinterpret_cast<ulonglong2*>(S.stage);
    const int nrec = (cnt + 1) >> 1;
    if (lane < nrec) {
      const bool two = lane + nrec < cnt;
      const uint32_t n0 = ring[lane], n1 = two ? ring[lane + nrec] : n0;
      double x0, y0, z0, m0, x1, y1, z1, m1;  // m: the mass and the first quadrupole term
      ld32(a.src + n0, x0, y0, z0, m0);
      ld32(a.src + n1, x1, y1, z1, m1);
      float q0[8], q1[8];
      if (QUAD) {
        ld32(reinterpret_cast<const char*>(a.src + n0) + 32, q0);
        ld32(reinterpret_cast<const char*>(a.src + n1) + 32, q1);
      }
      const double scale = S.scale;
      f2 px = offsets(x0, x1, S.centre[0], scale), py = offsets(y0, y1, S.centre[1], scale);
      f2 pz = offsets(z0, z1, S.centre[2], scale);
      if (!two) {
        px = f2_pack(__uint_as_float((uint32_t)px), kFarAway), m1 = 0.0;
#pragma unroll
        for (int k = 0; k < 5; ++k) q1[k] = 0.f;
      }
      rec[lane] = make_ulonglong2(px, py);
      rec[kCellPlane + lane] =
          make_ulonglong2(pz, f2_pack(__int_as_float(__double2loint(m0)), __int_as_float(__double2loint(m1))));
      if (QUAD) {
        const float s2 = -(float)S.scale2;
        const f2 n2 = f2_pack(s2, s2);  // the quadrupoles negated, in scaled units
        rec[2 * kCellPlane + lane] =
            make_ulonglong2(f2_mul(f2_pack(__int_as_float(__double2hiint(m0)), __int_as_float(__double2hiint(m1))), n2),
                            f2_mul(f2_pack(q0[0], q1[0]), n2));
        rec[3 * kCellPlane + lane] = make_ulonglong2(f2_mul(f2_pack(q0[1], q1[1]), n2), f2_mul(f2_pack(q0[2], q1[2]), n2));
        rec[4 * kCellPlane + lane] = make_ulonglong2(f2_mul(f2_pack(q0[3], q1[3]), n2), f2_mul(f2_pack(q0[4], q1[4]), n2));
      }
    }
    __syncwarp();
    const f2 e2 = twice(S.eps2);
    for (int s = first; s < nrec; s += ng) {
      const ulonglong2 xy = rec[s], zm = rec[kCellPlane + s];
      ulonglong2 n01 = {}, n23 = {}, n45 = {};
      if (QUAD) n01 = rec[2 * kCellPlane + s], n23 = rec[3 * kCellPlane + s], n45 = rec[4 * kCellPlane + s];
      cell_body(xy, zm, n01, n23, n45, e2, t0x, t0y, t0z, a0x, a0y, a0z);
      cell_body(xy, zm, n01, n23, n45, e2, t1x, t1y, t1z, a1x, a1y, a1z);
    }
    pend += (nrec + ng - 1) * inv_ng >> 16;
    if (pend >= kFlushTerms) flush();
    __syncwarp();
  }

  // direct particles: particle indices ring[0 .. cnt), cnt <= kPartBatch
  __device__ __forceinline__ void parts(const uint32_t* ring, int cnt) {
    ulonglong2* rec = reinterpret_cast<ulonglong2*>(S.stage);
    const int nrec = (cnt + 1) >> 1;
    for (int r = lane; r < nrec; r += 32) {
      const bool two = r + nrec < cnt;
      const uint32_t n0 = ring[r], n1 = two ? ring[r + nrec] : n0;
      double x0, y0, z0, m0, x1, y1, z1, m1;
      ld32(a.pm + n0, x0, y0, z0, m0);
      ld32(a.pm + n1, x1, y1, z1, m1);
      const double scale = S.scale;
      f2 px = offsets(x0, x1, S.centre[0], scale), py = offsets(y0, y1, S.centre[1], scale);
      f2 pz = offsets(z0, z1, S.centre[2], scale);
      if (!two) px = f2_pack(__uint_as_float((uint32_t)px), kFarAway);
      rec[r] = make_ulonglong2(px, py);
      rec[kPartPlane + r] = make_ulonglong2(pz, f2_pack((float)m0, two ? (float)m1 : 0.f));
    }
    __syncwarp();
    const f2 e2 = twice(S.eps2);
    for (int s = first; s < nrec; s += ng) {
      const ulonglong2 xy = rec[s], zm = rec[kPartPlane + s];
      part_body(xy, zm, e2, t0x, t0y, t0z, a0x, a0y, a0z);
      part_body(xy, zm, e2, t1x, t1y, t1z, a1x, a1y, a1z);
    }
    pend += (nrec + ng - 1) * inv_ng >> 16;
    if (pend >= kFlushTerms) flush();
    __syncwarp();
  }

  // After a list: the lane groups' sums, added in group order into the
  // targets' FP64 sums out[0 .. n).
  __device__ __forceinline__ void finish(int n, double (*out)[3]) {
    if (pend) flush();
    __syncwarp();
    add_group_sums(S, lane, n, (n + 1) >> 1, ng, out);
  }
};

// Plain FP64: the same lane layout and lists; absolute positions, the formula
// of accel_from_source with multiplications by 1/r^2 in place of its
// divisions.
template <bool QUAD, bool MASK>
struct F64Eval {
  static constexpr int kCellBatch = 32, kPartBatch = 64;
  static constexpr int kBlocksPerSm = 4;
  // planes of double2 per source: (x, y) (z, m) (q0, q1) (q2, q3) (q4, q5)
  static_assert(5 * 16 * kCellBatch <= kStageBytes && 2 * 16 * kPartBatch <= kStageBytes && kPartBatch + 31 < kRing,
                "batches too large");
  const WalkArgs& a;
  WarpSmem& S;
  int lane, ng, first;
  double t0x, t0y, t0z, t1x, t1y, t1z;
  double a0x, a0y, a0z, a1x, a1y, a1z;

  __device__ F64Eval(const WalkArgs& args, WarpSmem& S_, int lane_, double eps2_)
      : a(args), S(S_), lane(lane_) {
    S.eps2 = eps2_;
  }

  __device__ void setup(uint32_t p0, int n, double, double, double) {
    const int lpg = (n + 1) >> 1, inv = 65536 / lpg + 1;
    const int g = lane * inv >> 16, t0 = lane - g * lpg, t1 = t0 + lpg < n ? t0 + lpg : t0;
    ng = 32 * inv >> 16;
    first = g < ng ? g : 1 << 30;
    const double4 q0 = a.pm[p0 + t0], q1 = a.pm[p0 + t1];
    t0x = q0.x, t0y = q0.y, t0z = q0.z;
    t1x = q1.x, t1y = q1.y, t1z = q1.z;
    a0x = a0y = a0z = a1x = a1y = a1z = 0.0;
  }

  __device__ __forceinline__ void cell_body(double2 xy, double2 zm, double2 q01, double2 q23, double2 q45, double eps2,
                                            double tx, double ty, double tz, double& ax, double& ay, double& az) const {
    const double dx = xy.x - tx, dy = xy.y - ty, dz = zm.x - tz;
    const double r2 = dx * dx + dy * dy + dz * dz + eps2;
    double ri = rsqrt(r2);
    if (!QUAD && MASK) ri = r2 > 0.0 ? ri : 0.0;
    const double ri2 = ri * ri;
    const double ri3 = ri * ri2;
    if (QUAD) {
      const double qx = q01.x * dx + q23.y * dy + q45.x * dz;
      const double qy = q23.y * dx + q01.y * dy + q45.y * dz;
      const double qz = q45.x * dx + q45.y * dy + q23.x * dz;
      const double dqd = dx * qx + dy * qy + dz * qz;
      const double ri5 = ri3 * ri2;
      const double c = zm.y * ri3 + 2.5 * dqd * (ri5 * ri2);
      ax += c * dx - ri5 * qx;
      ay += c * dy - ri5 * qy;
      az += c * dz - ri5 * qz;
    } else {
      const double c = zm.y * ri3;
      ax += c * dx, ay += c * dy, az += c * dz;
    }
  }

  __device__ __forceinline__ void part_body(double2 xy, double2 zm, double eps2, double tx, double ty, double tz, double& ax,
                                            double& ay, double& az) const {
    const double dx = xy.x - tx, dy = xy.y - ty, dz = zm.x - tz;
    const double r2 = dx * dx + dy * dy + dz * dz + eps2;
    double ri = rsqrt(r2);
    if (MASK) ri = r2 > 0.0 ? ri : 0.0;
    const double c = zm.y * (ri * ri) * ri;
    ax += c * dx, ay += c * dy, az += c * dz;
  }

  __device__ __forceinline__ void cells(const uint32_t* ring, int cnt) {
    double2* rec = reinterpret_cast<double2*>(S.stage);
    if (lane < cnt) {
      const uint32_t n = ring[lane];
      double x, y, z, m;
      ld32(a.mom + n, x, y, z, m);
      rec[lane] = make_double2(x, y), rec[kCellBatch + lane] = make_double2(z, m);
      if (QUAD) {
        // traceless Q = 3 I - tr(I) delta (accel_from_source, multipole.h:185-188)
        const double2* ip = reinterpret_cast<const double2*>(a.iab + (size_t)n * 6);
        const double2 i01 = ip[0], i23 = ip[1], i45 = ip[2];
        const double tr = __dadd_rn(__dadd_rn(i01.x, i01.y), i23.x);
        rec[2 * kCellBatch + lane] =
            make_double2(__dsub_rn(__dmul_rn(3.0, i01.x), tr), __dsub_rn(__dmul_rn(3.0, i01.y), tr));
        rec[3 * kCellBatch + lane] = make_double2(__dsub_rn(__dmul_rn(3.0, i23.x), tr), __dmul_rn(3.0, i23.y));
        rec[4 * kCellBatch + lane] = make_double2(__dmul_rn(3.0, i45.x), __dmul_rn(3.0, i45.y));
      }
    }
    __syncwarp();
    const double e2 = S.eps2;
    for (int s = first; s < cnt; s += ng) {
      const double2 xy = rec[s], zm = rec[kCellBatch + s];
      double2 q01 = {}, q23 = {}, q45 = {};
      if (QUAD) q01 = rec[2 * kCellBatch + s], q23 = rec[3 * kCellBatch + s], q45 = rec[4 * kCellBatch + s];
      cell_body(xy, zm, q01, q23, q45, e2, t0x, t0y, t0z, a0x, a0y, a0z);
      cell_body(xy, zm, q01, q23, q45, e2, t1x, t1y, t1z, a1x, a1y, a1z);
    }
    __syncwarp();
  }

  __device__ __forceinline__ void parts(const uint32_t* ring, int cnt) {
    double2* rec = reinterpret_cast<double2*>(S.stage);
    for (int i = lane; i < cnt; i += 32) {
      double x, y, z, m;
      ld32(a.pm + ring[i], x, y, z, m);
      rec[i] = make_double2(x, y), rec[kPartBatch + i] = make_double2(z, m);
    }
    __syncwarp();
    const double e2 = S.eps2;
    for (int s = first; s < cnt; s += ng) {
      const double2 xy = rec[s], zm = rec[kPartBatch + s];
      part_body(xy, zm, e2, t0x, t0y, t0z, a0x, a0y, a0z);
      part_body(xy, zm, e2, t1x, t1y, t1z, a1x, a1y, a1z);
    }
    __syncwarp();
  }

  __device__ __forceinline__ void finish(int n, double (*out)[3]) {
    S.sums[0][lane] = a0x, S.sums[1][lane] = a0y, S.sums[2][lane] = a0z;
    S.sums[3][lane] = a1x, S.sums[4][lane] = a1y, S.sums[5][lane] = a1z;
    __syncwarp();
    add_group_sums(S, lane, n, (n + 1) >> 1, ng, out);
  }
};

// ---------------------------------------------------------------------------
// The shared walk of a group of k <= kMaxTargets targets, in the spirit of
// GroupWalker::visit (grouped_ttg.h:204-289) taken to every level: one
// traversal from the root whose stack entries (runs of sibling nodes) carry
// the mask of targets that still need them.  Each popped node is first tested
// against the group's particle box: accepted there (mac_accept_bbox) ->
// accepted by every target in the mask; rejected for every point of it
// (mac_reject_all, multipole.h:158-160) -> opened by every target in the
// mask; otherwise each target tests its own box: lane t + k * r holds target
// t's box and tests the r-th of the 32 / k nodes taken at a time.  A node
// taken by every target of the group goes to the dense list, one taken by
// some to the partial list with its mask; opened interior nodes push their
// children with the mask of the targets that opened them.  Every target's
// list is exactly what a walk of its own box from the root gives
// (multipole.h's tests are monotone in the box).
// The traversal only writes lists.  Without the evaluators' registers and
// queues beside it the kernel runs 24 warps per SM (80 registers, 9.3 KB of
// shared memory per warp) instead of 16, and each part is a loop of its own:
// walk per evaluation 30.5 to 23.2 ms at 4M, 7.39 to 5.80 at 1M, 1.89 to 1.46
// at 262k (leaf 16, theta 0.5); in FP64 12.8 to 9.5 ms at 1M.  With 5 blocks
// of 4 warps per SM 23.8 ms at 4M, with 4 25.1.

// The tests run in FP32 first, on offsets from the group's centre in the
// system's units.  With u = 2^-24 and M the largest coordinate of the node and
// of the group's box, an offset to a box face is off by at most E = 4 u M, and
// a squared distance v by at most 2 sqrt(3 v) E + 3 E^2 (and a few u v), which
// is at most 2^-14 v + 3 E^2 (1 + 2^14), and 3 E^2 (1 + 2^14) < 4e-9 M^2.  So with K =
// 4e-9 M^2 (+ 1e-30, far below any edge^2, for the range FP32 loses) a node
// is certainly accepted when v > accept = (edge^2 / theta^2 + K) / (1 - 2^-14)
// and certainly not when v < reject = (edge^2 / theta^2 - K) / (1 + 2^-14), both
// factors with 2e-5 to spare for the rounding of the terms themselves; NaN and
// infinity leave both false.  What lies between - one test in some thousands -
// is decided by the FP64 test, so every decision is the reference's.
// Walk with them / with the FP64 tests alone: 20.7 / 21.4 ms at 4M, 5.17 /
// 5.37 at 1M, 2.09 / 2.18 with monopoles (traversal instructions 0.63e9 of 0.84e9).

__device__ __forceinline__ float near2f(const float lo[3], const float hi[3], float x, float y, float z) {
  const float dx = fmaxf(fmaxf(lo[0] - x, x - hi[0]), 0.f);
  const float dy = fmaxf(fmaxf(lo[1] - y, y - hi[1]), 0.f);
  const float dz = fmaxf(fmaxf(lo[2] - z, z - hi[2]), 0.f);
  return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

__device__ __forceinline__ float far2f(const float lo[3], const float hi[3], float x, float y, float z) {
  const float dx = fmaxf(x - lo[0], hi[0] - x);
  const float dy = fmaxf(y - lo[1], hi[1] - y);
  const float dz = fmaxf(z - lo[2], hi[2] - z);
  return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

// prog: where to publish the cells written so far (a dense job evaluates
// them meanwhile), or null.
// Returns true when a list may be too full for another step (the lists are
// then to be taken and reset, and the traversal goes on where it stopped).
template <bool PAIRS>
__device__ __forceinline__ bool traverse(const WalkArgs& a, WarpSmem& S, double theta2, uint2* __restrict__ dl,
                                         uint2* __restrict__ pl, uint32_t* prog, int lane) {
  const uint32_t k = S.job.k;
  Walk w = S.job.w;
  const uint32_t lt = lanemask_lt();
  const uint32_t full = (1u << k) - 1u;  // k <= kMaxTargets < 32
  StepScratch& X = *reinterpret_cast<StepScratch*>(S.stage);
  const uint32_t per = 32u / k, sub = (uint32_t)lane / k, tgt = (uint32_t)lane - sub * k;
  const double gx = 0.5 * (S.glo[0] + S.ghi[0]), gy = 0.5 * (S.glo[1] + S.ghi[1]), gz = 0.5 * (S.glo[2] + S.ghi[2]);
  float lo[3], hi[3], glo[3], ghi[3], reach = 0.f;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double c = d == 0 ? gx : d == 1 ? gy : gz, sc = S.scale;
    lo[d] = (float)((S.tlo[tgt][d] - c) * sc), hi[d] = (float)((S.thi[tgt][d] - c) * sc);
    glo[d] = (float)((S.glo[d] - c) * sc), ghi[d] = (float)((S.ghi[d] - c) * sc);
    reach = fmaxf(reach, fmaxf(fabsf(glo[d]), fabsf(ghi[d])));
  }
  const float inv_theta2 = (float)(1.0 / theta2);
  const uint32_t max_steps = a.st->n_nodes + 2;  // a walk pops each node at most once
  S.job.told = 0u;
  bool more = false;
  while (w.top) {
    if (w.ndc + w.ndr + 32 > kDenseCap || w.npc + w.npr + 64 > kListCap) {
      more = true;
      break;
    }
    if (++w.steps > max_steps) {  // a corrupt tree
      if (lane == 0) atomicOr(&a.st->status, kStWalkLimit);
      w.top = 0;
      break;
    }
    // pop up to 32 nodes off the top runs: lane i looks at the i-th run from the top
    const uint32_t have = min(w.top, 32u);
    uint2 ent = make_uint2(0u, 0u);
    if ((uint32_t)lane < have) ent = S.stack[w.top - 1 - lane];
    const uint32_t c = ent.y >> 24;
    const uint32_t inc = warp_incl_scan_u32(c, lane), excl = inc - c;
    const uint32_t room = (uint32_t)kStackCap - (kLevels + 1);
    uint32_t n = min(__shfl_sync(kFull, inc, 31), 32u);
    n = min(n, w.top < room ? room - w.top : 1u);
    // the run holding node slot `lane`: the runs' first slots as bits, counted up to the lane
    const uint32_t heads = __reduce_or_sync(kFull, (c && excl < 32u) ? 1u << excl : 0u);
    const uint32_t run = (uint32_t)__popc(heads & (lt | (1u << lane))) - 1u;
    const uint32_t node = __shfl_sync(kFull, ent.x - excl, run) + (uint32_t)lane;
    const uint32_t mask = __shfl_sync(kFull, ent.y, run) & kMaskBits;
    const bool valid = (uint32_t)lane < n;
    const uint32_t done = (uint32_t)__popc(__ballot_sync(kFull, c && inc <= n));
    __syncwarp();
    if (c && excl < n && n < inc) S.stack[w.top - 1 - lane] = make_uint2(ent.x + (n - excl), ent.y - ((n - excl) << 24));
    w.top -= done;
    uint2 link = make_uint2(0u, 0u);  // first child and children, or first particle and particles | kLeafBit
    float x = 0.f, y = 0.f, z = 0.f, accept = 0.f, reject = 0.f;
    bool acc = false, rej = false;
    if (valid) {
      double4 c4;
      ld32(a.wcom + node, c4.x, c4.y, c4.z, c4.w);  // com xyz, edge^2
      link = a.wlink[node];
      const double sc = S.scale;
      x = (float)((c4.x - gx) * sc), y = (float)((c4.y - gy) * sc), z = (float)((c4.z - gz) * sc);
      const float m = fmaxf(fmaxf(fabsf(x), fabsf(y)), fmaxf(fabsf(z), reach));
      const float slack = fmaf(4.0e-9f * m, m, 1.0e-30f), q = (float)(c4.w * S.scale2) * inv_theta2;
      accept = (q + slack) * 1.00008f, reject = (q - slack) * 0.99992f;
      const float n2 = near2f(glo, ghi, x, y, z);
      acc = n2 > accept;
      // mac_accept_bbox: theta^2 * near^2 > edge^2 (multipole.h:151-153)
      if (!acc && !(n2 < reject)) acc = __dmul_rn(theta2, near2(S.glo, S.ghi, c4.x, c4.y, c4.z)) > c4.w;
      if (!acc) {
        // one target: its box is the group's, so not accepted means opened
        const float f2v = far2f(glo, ghi, x, y, z);
        rej = k == 1 || f2v < reject;
        if (!rej && !(f2v > accept)) rej = __dmul_rn(theta2, far2(S.glo, S.ghi, c4.x, c4.y, c4.z)) <= c4.w;
      }
    }
    uint32_t A = acc ? mask : 0u, O = rej ? mask : 0u;
    // undecided nodes: every target tests its own box
    const bool und = valid && !acc && !rej;
    const uint32_t um = __ballot_sync(kFull, und);
    if (um) {
      const uint32_t rank = (uint32_t)__popc(um & lt), nu = (uint32_t)__popc(um);
      if (und) X.node[rank] = make_float4(x, y, z, accept), X.reject[rank] = reject, X.id[rank] = node;
      __syncwarp();
      for (uint32_t base = 0; base < nu; base += per) {
        const uint32_t e = base + sub;
        bool ok = false;
        if (sub < per && e < nu) {
          const float4 q = X.node[e];
          const float n2 = near2f(lo, hi, q.x, q.y, q.z);
          ok = n2 > q.w;
          if (!ok && !(n2 < X.reject[e])) {
            double4 c4;
            ld32(a.wcom + X.id[e], c4.x, c4.y, c4.z, c4.w);
            ok = __dmul_rn(theta2, near2(S.tlo[tgt], S.thi[tgt], c4.x, c4.y, c4.z)) > c4.w;
          }
        }
        const uint32_t bits = __ballot_sync(kFull, ok);
        if (tgt == 0 && sub < per && e < nu) X.accepts[e] = (bits >> (sub * k)) & full;
      }
      __syncwarp();
      if (und) A = X.accepts[rank] & mask, O = mask & ~A;
    }
    const bool leaf = (link.y & kLeafBit) != 0u;
    const uint32_t cnt = link.y & ~kLeafBit;
    // cells every target takes, some take
    const bool dc = A != 0u && A == full, pc = A != 0u && A != full;
    uint32_t m = __ballot_sync(kFull, dc);
    if (dc) dl[w.ndc + __popc(m & lt)] = make_uint2(node, 1u);
    w.ndc += __popc(m);
    if (PAIRS && prog && w.ndc - S.job.told >= 64) {  // the dense job may take them
      __threadfence();
      __syncwarp();
      if (lane == 0) st_volatile(prog, w.ndc);
      S.job.told = w.ndc;
    }
    m = __ballot_sync(kFull, pc);
    if (pc) pl[w.npc + __popc(m & lt)] = make_uint2(node, A);
    w.npc += __popc(m);
    // leaves every target opens, some open
    const bool dr = leaf && O == full, pr = leaf && O != 0u && O != full;
    m = __ballot_sync(kFull, dr);
    if (dr) dl[kDenseCap - 1u - (w.ndr + __popc(m & lt))] = make_uint2(link.x, cnt);
    w.ndr += __popc(m);
    m = __ballot_sync(kFull, pr);
    if (pr)
      pl[kListCap - 1u - (w.npr + __popc(m & lt))] =
          cnt < kByNode ? make_uint2(link.x, O | (cnt << kCountShift)) : make_uint2(node, O | (kByNode << kCountShift));
    w.npr += __popc(m);
    // opened interior nodes: their children, with the targets that opened them
    const bool in = O != 0u && !leaf;
    m = __ballot_sync(kFull, in);
    if (in) S.stack[w.top + __popc(m & lt)] = make_uint2(link.x, O | (cnt << 24));
    w.top += __popc(m);
    __syncwarp();
  }
  S.job.w = w;
  return more;
}

// Entries i and i + 1 of a list of n, at p.
__device__ __forceinline__ uint4 load_pair(const uint4* p, uint32_t i, uint32_t n) {
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (i < n) v = *p;
  if (i + 1 >= n) v.w = 0u;
  return v;
}

// A dense job's wait (bounded, as wait_lengths) for cells beyond `at` (a
// multiple of 64) in its group's progress word: the word, or kAborted after
// `limit` polls.  The group's target jobs, which wait for this one, are then
// told (kListLost): each would poll to its own limit, half a second.
__device__ __forceinline__ uint32_t wait_cells(const uint32_t* prog, uint32_t* length, uint32_t at, int limit,
                                               DevState* st, int lane) {
  for (int spins = 0;; ++spins) {
    uint32_t v = ld_volatile(prog);
    v = __shfl_sync(kFull, v == kListPending ? 0u : v, 0);
    if ((v & (kFinal | kAborted)) || (v & ~63u) > at) return v;
    if (spins >= limit) {
      if (lane == 0) {
        atomicOr(&st->status, kStSpinLimit);
        st_volatile(length, kListLost);
      }
      return kAborted;
    }
    __nanosleep(64);
  }
}

// Both waits on prepared words (bhg_selftest_walk_wait), one warp: a group's
// progress and its list length, and another group's list length.  out: the
// progress, the first length as that wait left it, the second length.
__global__ void k_walk_wait_probe(uint32_t* words, int limit, DevState* st, uint32_t* out) {
  const int lane = threadIdx.x & 31;
  const uint32_t cells = wait_cells(words, words + 1, 64u, limit, st, lane);
  const uint32_t len = wait_lengths(words + 2, limit, st, lane);
  if (lane == 0) out[0] = cells, out[1] = ld_volatile(words + 1), out[2] = len;
}

void launch_walk_wait_probe(uint32_t* words, int limit, DevState* st, uint32_t* out, cudaStream_t s) {
  k_walk_wait_probe<<<1, 32, 0, s>>>(words, limit, st, out);
}

// A dense job's further cells, beyond `at` (a multiple of 64): those that may
// be read, a multiple of 64 too unless they are all.
__device__ __forceinline__ uint32_t more_cells(const WalkArgs& a, WarpSmem& S, uint32_t at, int lane) {
  Job& J = S.job;
  const uint32_t v = wait_cells(a.prog + J.gi, a.gnl + J.gi, at, kSpinLimit, a.st, lane);
  __threadfence();  // the cells after the word
  if (!(v & (kFinal | kAborted))) return v & ~63u;
  __syncwarp();
  J.poll = 0u;
  J.aborted = v & kAborted ? 1u : 0u;
  J.w.ndc = J.aborted ? at : v & 0xfffu;
  J.w.ndr = J.aborted ? 0u : (v >> 12) & 0xfffu;
  __syncwarp();
  return J.w.ndc;
}

// Evaluates the entries of the job's dense or partial list that `sel` picks
// (bits of the entry's second word) on the evaluator's tn targets: first the
// cells, then the runs.  Windows of 64 cells or 32 runs, the next one loaded
// while the current one is used, fill a ring; full batches of it are evaluated.
template <bool PAIRS, class E>
__device__ __forceinline__ void list_pass(E& ev, const WalkArgs& a, WarpSmem& S, bool dense, uint32_t sel, uint32_t tn,
                                          int lane) {
  const uint32_t lt = lanemask_lt();
  uint32_t at = 0, held = 0;
  // two entries per lane and window (16-byte loads; the list's end is read as
  // entries that nothing picks)
  const uint4* pairs = reinterpret_cast<const uint4*>(dense ? S.job.dense : S.job.partial) + lane;
  uint32_t nc = dense ? S.job.w.ndc : S.job.w.npc;
  uint4 next = load_pair(pairs, 2u * lane, nc);
  for (;;) {
    while (held < (uint32_t)E::kCellBatch) {
      if (at >= nc) {
        if (!PAIRS || !S.job.poll) break;
        nc = more_cells(a, S, at, lane);
        next = load_pair(pairs, at + 2u * lane, nc);
        continue;
      }
      const uint4 e = next;
      at += 64;
      pairs += 32;
      next = load_pair(pairs, at + 2u * lane, nc);
      const bool h0 = (e.y & sel) != 0u, h1 = (e.w & sel) != 0u;
      const uint32_t m0 = __ballot_sync(kFull, h0), m1 = __ballot_sync(kFull, h1);
      const uint32_t pos = held + __popc(m0 & lt) + __popc(m1 & lt);
      if (h0) S.ring[pos] = e.x;
      if (h1) S.ring[pos + (h0 ? 1u : 0u)] = e.z;
      held += __popc(m0) + __popc(m1);
    }
    if (!held) break;
    __syncwarp();
    const uint32_t cnt = min(held, (uint32_t)E::kCellBatch);
    ev.cells(S.ring, (int)cnt);
    if (lane == 0) S.ncell += cnt * tn;
    held -= cnt;
    if (held) {  // at most kCellBatch - 1 + 64 - kCellBatch = 63 are left
      const uint32_t v0 = S.ring[cnt + lane], v1 = S.ring[cnt + 32 + lane];
      __syncwarp();
      if ((uint32_t)lane < held) S.ring[lane] = v0;
      if ((uint32_t)lane + 32 < held) S.ring[lane + 32] = v1;
    }
  }
  // runs: the particles of the picked runs of a window, 32 at a time
  const uint2* back = dense ? S.job.dense + kDenseCap - 1 : S.job.partial + kListCap - 1;
  const uint32_t nr = dense ? S.job.w.ndr : S.job.w.npr;
  at = 0;
  uint2 ahead = (uint32_t)lane < nr ? back[-lane] : make_uint2(0u, 0u);
  uint32_t tot = 0, base = 0, before = 0, cnt = 0, excl = 0;
  for (;;) {
    while (held < (uint32_t)E::kPartBatch) {
      if (base < tot) {
        // the run holding particle base + lane: first particles as bits
        const uint32_t heads =
            __reduce_or_sync(kFull, (cnt && excl >= base && excl < base + 32u) ? 1u << (excl - base) : 0u);
        const uint32_t run = before + (uint32_t)__popc(heads & (lt | (1u << lane))) - 1u;
        const uint32_t take = min(32u, tot - base);
        if ((uint32_t)lane < take) S.ring[held + lane] = S.delta[run] + base + (uint32_t)lane;
        before += __popc(heads);
        held += take;
        base += 32u;
        continue;
      }
      if (at >= nr) break;
      uint2 e = ahead;
      at += 32;
      const uint32_t j = at + (uint32_t)lane;
      ahead = j < nr ? back[-(int)j] : make_uint2(0u, 0u);
      const bool hit = (e.y & sel) != 0u;
      const uint32_t m = __ballot_sync(kFull, hit);
      if (!m) continue;
      cnt = hit ? (dense ? e.y : e.y >> kCountShift) : 0u;
      if (!dense && cnt == kByNode) {
        const uint2 link = a.wlink[e.x];
        e.x = link.x, cnt = link.y & ~kLeafBit;
      }
      const uint32_t inc = warp_incl_scan_u32(cnt, lane);
      excl = inc - cnt;
      tot = __shfl_sync(kFull, inc, 31);
      base = before = 0;
      __syncwarp();
      if (hit) S.delta[__popc(m & lt)] = e.x - excl;
      __syncwarp();
    }
    if (!held) break;
    __syncwarp();
    const uint32_t c = min(held, (uint32_t)E::kPartBatch);
    ev.parts(S.ring, (int)c);
    if (lane == 0) S.npart += c * tn;
    held -= c;
    if (held) {
      const uint32_t v = S.ring[c + lane];
      __syncwarp();
      if ((uint32_t)lane < held) S.ring[lane] = v;
    }
  }
}

// The targets' particle ranges and boxes and the group's box; returns the
// group's particles.
__device__ __forceinline__ uint32_t group_boxes(const WalkArgs& a, WarpSmem& S, int lane) {
  const Job& g = S.job;
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  uint32_t tb = 0, tc = 0;
  if ((uint32_t)lane < g.k) {
    const uint32_t tn = a.targets[g.t0 + lane];
    tb = a.nbegin[tn], tc = a.ncount[tn];
    S.tbeg[lane] = tb, S.tcnt[lane] = tc;
  }
  const uint32_t n = __shfl_sync(kFull, tb + tc, (int)g.k - 1) - g.p0;
  if (n > (uint32_t)kGroupMax) {  // one large target
    particle_box(a.pm, g.p0, n, lane, lo, hi);
  } else {
    double (*pos)[3] = reinterpret_cast<double (*)[3]>(S.stage);
    for (uint32_t i = lane; i < n; i += 32) {
      const double4 q = a.pm[g.p0 + i];
      pos[i][0] = q.x, pos[i][1] = q.y, pos[i][2] = q.z;
    }
    __syncwarp();
    for (uint32_t i = 0; i < tc; ++i) {
      const double* q = pos[tb - g.p0 + i];
#pragma unroll
      for (int d = 0; d < 3; ++d) lo[d] = fmin(lo[d], q[d]), hi[d] = fmax(hi[d], q[d]);
    }
  }
  if ((uint32_t)lane < g.k) {
#pragma unroll
    for (int d = 0; d < 3; ++d) S.tlo[lane][d] = lo[d], S.thi[lane][d] = hi[d];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      lo[d] = fmin(lo[d], __shfl_xor_sync(kFull, lo[d], o));
      hi[d] = fmax(hi[d], __shfl_xor_sync(kFull, hi[d], o));
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int d = 0; d < 3; ++d) S.glo[d] = lo[d], S.ghi[d] = hi[d];
  }
  __syncwarp();
  return n;
}

// One warp per walk group (a run of targets, k_pack_groups): the group's
// traversal writes its lists, then list passes evaluate them - pass 0 the
// dense list on all the group's particles, pass 1 + i the partial list's
// entries that target i takes on that target's particles, each pass adding
// its part onto the group's FP64 sums - and the kick/drift follows.  When a
// list fills up, the traversal pauses: that list's passes run (pass 0, or
// all), and it goes on with the list empty.  A group of one target larger
// than kGroupMax particles is walked once per kGroupMax of its particles.
//
// With few groups (n_groups <= a.nslots: about as many as warps, so the
// largest group's targets would set the kernel's time) the work is cut in
// two: the warps first take the groups' traversals and dense passes (and the
// groups of one target whole), each leaving its group's FP64 sums and partial
// list in the group's slot and publishing the list's lengths; then they take
// every target's pass as a job of its own, starting as soon as the group's
// lengths are published.  With fewer groups still (two warps for each), a
// group's dense pass is a job of its own too, which takes the cells while the
// traversal finds them; if that has to pause, it evaluates its lists itself and
// goes on in another dense list (dense_slot).  A job waits only for jobs
// handed out before it, which running warps hold and which wait for none or
// for such jobs, so every wait ends; a wait is still bounded (kStSpinLimit,
// the job skipped).  All schedules run the same passes on the same batches and
// add their parts in the same order, so the results are the same bits.  Walk with / without dense jobs: 0.25 / 0.34 ms
// at 16k, 0.42 / 0.56 at 65k, 0.63 / 0.72 at 40k in FP64.
template <class E, bool QUAD, bool PAIRS>
__global__ void __launch_bounds__(kWalkThreads, E::kBlocksPerSm) k_walk(WalkArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WarpSmem& S = reinterpret_cast<WarpSmem*>(smem_raw)[warp];
  if (a.st->status & (kStNonFinite | kStNodeOverflow | kStSpinLimit)) return;  // the build failed: touch nothing
  Job& J = S.job;
  if (lane == 0) S.ncell = S.npart = 0ull;
  J.kind = kWholeJob;
  for (;;) {
    const uint32_t ngroups = a.st->n_groups, ntargets = a.st->n_targets;
    const bool two_pass = ngroups <= a.nslots, paired = PAIRS && two_pass && 2 * ngroups <= gridDim.x * kWalkWarps;
    uint32_t next = 0;
    if (lane == 0) next = atomicAdd(J.kind == kTargetJob ? &a.st->walk_next2 : &a.st->walk_next, 1u);
    next = __shfl_sync(kFull, next, 0);
    __syncwarp();  // every lane is done with the last job
    if (J.kind == kTargetJob) {
      if (next >= ntargets) break;
      // its group: the last whose first target is at or before it
      uint32_t gi = 0, hi = ngroups;
      while (hi - gi > 1) {
        const uint32_t mid = (gi + hi) >> 1;
        if (a.groups[mid] <= next) gi = mid;
        else hi = mid;
      }
      J.gi = gi, J.ti = next;
    } else if (next < ngroups) {
      J.gi = next;
    } else if (paired && next < 2 * ngroups) {
      __syncwarp();
      J.gi = next - ngroups, J.kind = kDenseJob;
    } else if (two_pass) {
      __syncwarp();  // every lane has read the kind
      J.kind = kTargetJob;
      continue;
    } else {
      break;
    }
    {
      const GroupInfo g = group_info(a, J.gi, ngroups, ntargets);
      J.t0 = g.t0, J.k = g.k, J.p0 = g.p0, J.sys = g.s;
    }
    if (walked_elsewhere(a, J.sys)) continue;
    if (J.kind != kWholeJob && J.k == 1) continue;  // done whole by its group
    J.w = Walk{0u, 0u, 0u, 0u, 0u, 0u};
    set_units(S, a.sys[J.sys].hw);
    // the partial list is the warp's or (two-pass schedule) the group's, the
    // dense one the warp's or (with dense jobs) the group's
    const size_t wid = (size_t)blockIdx.x * kWalkWarps + warp;
    J.dense = a.dlist + dense_slot(paired, false, J.gi, ngroups, wid) * kDenseCap;
    J.partial = a.wlist + (two_pass ? (size_t)J.gi : wid) * kListCap;
    J.poll = J.kind == kDenseJob;
    J.aborted = 0u;
    if (J.kind == kTargetJob) {
      const uint32_t len = wait_lengths(a.gnl + J.gi, kSpinLimit, a.st, lane);
      if (len == kListLost) continue;
      __threadfence();  // the group's sums and list after its lengths
      J.w.npc = len & 0xffffu, J.w.npr = len >> 16;
      const uint32_t bit = J.ti - J.t0, tn = a.targets[J.ti];
      const uint32_t tb = a.nbegin[tn], tc = a.ncount[tn];  // tc <= kGroupMax: inside a group
      double lo[3], hi[3];
      particle_box(a.pm, tb, tc, lane, lo, hi);
      S.tbeg[bit] = tb, S.tcnt[bit] = tc;
#pragma unroll
      for (int d = 0; d < 3; ++d) S.tlo[bit][d] = lo[d], S.thi[bit][d] = hi[d];
      const double* gs = a.gsum + (size_t)J.gi * (kGroupMax * 3) + 3 * (tb - J.p0);
      for (uint32_t i = lane; i < 3 * tc; i += 32) (&S.acc[tb - J.p0][0])[i] = gs[i];
      J.n = tc;
      J.pass1 = 1 + bit;
      __syncwarp();
    } else {
      J.n = group_boxes(a, S, lane);
      J.pass1 = 0u;
      if (lane == 0) S.kept[0] = S.ncell, S.kept[1] = S.npart;
    }
    for (uint32_t b0 = 0; b0 < J.n; b0 += kGroupMax) {  // once, but for a large target
      J.b0 = b0;
      if (J.kind != kTargetJob) {
        for (uint32_t i = lane; i < 3 * kGroupMax; i += 32) (&S.acc[0][0])[i] = 0.0;
        // the traversal starts with the root
        S.stack[0] = make_uint2(a.sys[J.sys].root, ((1u << J.k) - 1u) | (1u << 24));
        J.w.top = 1, J.w.steps = 0;
        __syncwarp();
      }
      J.left = J.more = 0u;
      do {  // J.more is read at the end of a turn and written after the next one's traversal
        uint32_t pass = J.pass1;
        if (J.kind == kWholeJob) {
          const bool beside = paired && J.k > 1 && !J.aborted;  // a dense job evaluates beside
          const bool more =
              traverse<PAIRS>(a, S, a.prm[J.sys].theta2, J.dense, J.partial, beside ? a.prog + J.gi : nullptr, lane);
          if (beside) {
            if (!more && lane == 0) a.plen[J.gi] = J.w.npc | (J.w.npr << 16);
            __threadfence();  // the lists before the word
            __syncwarp();
            if (lane == 0) st_volatile(a.prog + J.gi, more ? kAborted : kFinal | (J.w.ndr << 12) | J.w.ndc);
            if (!more) {
              J.left = 1u;
              break;
            }
            J.aborted = 1u;
          }
          // all passes when the partial list is full or complete, else the dense one
          const bool all = more ? J.w.npc + J.w.npr + 64 > kListCap : !(two_pass && J.k > 1);
          J.more = more;
          pass = 0, J.pass1 = all && J.w.npc + J.w.npr ? J.k : 0u;
        }
        E ev(a, S, lane, a.prm[J.sys].eps2);
        for (; pass <= J.pass1; ++pass) {
          const bool dense = pass == 0;
          if ((dense ? J.w.ndc + J.w.ndr + J.poll : J.w.npc + J.w.npr) == 0) continue;
          const uint32_t i = pass - 1;
          const uint32_t tn = dense ? min(J.n - J.b0, (uint32_t)kGroupMax) : S.tcnt[i];
          {
            const double* lo = dense ? S.glo : S.tlo[i];
            const double* hi = dense ? S.ghi : S.thi[i];
            ev.setup(dense ? J.p0 + J.b0 : S.tbeg[i], (int)tn, 0.5 * (lo[0] + hi[0]), 0.5 * (lo[1] + hi[1]),
                     0.5 * (lo[2] + hi[2]));
          }
          list_pass<PAIRS>(ev, a, S, dense, dense ? kFull : 1u << i, tn, lane);
          ev.finish((int)tn, S.acc + (dense ? 0u : S.tbeg[i] - J.p0));
        }
        __syncwarp();
        J.w.ndc = J.w.ndr = 0;
        // the dense job may still be reading the list it was given
        if (paired && J.aborted) J.dense = a.dlist + dense_slot(true, true, J.gi, ngroups, wid) * kDenseCap;
        if (J.pass1) J.w.npc = J.w.npr = 0;
        __syncwarp();
      } while (J.more);
      if (J.left) continue;  // to the dense job
      if (J.kind == kDenseJob && J.aborted) {  // the group's own job evaluates its lists
        if (lane == 0) S.ncell = S.kept[0], S.npart = S.kept[1];
        continue;
      }
      const uint32_t nb = min(J.n - J.b0, (uint32_t)kGroupMax);
      if (two_pass && J.k > 1 && J.kind != kTargetJob) {  // leave the sums and the partial list to the target jobs
        double* gs = a.gsum + (size_t)J.gi * (kGroupMax * 3);
        for (uint32_t i = lane; i < 3 * nb; i += 32) gs[i] = (&S.acc[0][0])[i];
        __threadfence();  // the sums and the list before the lengths
        __syncwarp();
        if (lane == 0)
          st_volatile(a.gnl + J.gi, J.kind == kDenseJob ? __ldcg(a.plen + J.gi) : J.w.npc | (J.w.npr << 16));
      } else {
        const uint32_t off = J.kind == kTargetJob ? S.tbeg[J.ti - J.t0] - J.p0 : 0u;
        kick_drift(a, a.prm[J.sys], S.acc + off, J.p0 + off + J.b0, nb, lane);
      }
    }
  }
  if (lane == 0) {  // quad: cells are particle-cell interactions, else monopoles counted as particles
    atomicAdd(&a.st->pp, S.npart + (QUAD ? 0ull : S.ncell));
    atomicAdd(&a.st->pc, QUAD ? S.ncell : 0ull);
  }
}

template <class E, bool QUAD>
static void launch_one(const WalkArgs& a, uint32_t n, int grid, cudaStream_t s) {
  // Dense jobs pay from 4,096 particles on (with / without: 0.178 / 0.182 ms
  // there; 0.091 / 0.086 at 1,021, whose dense lists are too short to share
  // out).  Groups hold at most kGroupMax particles (or one large target, which
  // has no dense job): with more than this there are never two warps for
  // each, and the kernel without dense jobs is 0.6% faster.
  if (n >= 4096u && n <= (uint32_t)grid * kWalkWarps / 2 * kGroupMax)
    k_walk<E, QUAD, true><<<grid, kWalkThreads, kWalkSmem, s>>>(a);
  else k_walk<E, QUAD, false><<<grid, kWalkThreads, kWalkSmem, s>>>(a);
}

// Unsoftened split walks have a kernel of their own (bhg_walk_unsoftened.cu).
void launch_walk(const WalkArgs& a, uint32_t n, int precision, bool quad, bool mask, int grid, cudaStream_t s) {
  if (precision == 0) {
    if (mask) launch_walk_unsoftened(a, quad, grid, s);
    else quad ? launch_one<SplitEval<true>, true>(a, n, grid, s) : launch_one<SplitEval<false>, false>(a, n, grid, s);
  } else {
    if (quad) mask ? launch_one<F64Eval<true, true>, true>(a, n, grid, s) : launch_one<F64Eval<true, false>, true>(a, n, grid, s);
    else mask ? launch_one<F64Eval<false, true>, false>(a, n, grid, s) : launch_one<F64Eval<false, false>, false>(a, n, grid, s);
  }
}

template <class E, bool QUAD, bool PAIRS>
static int occ_of() {
  const auto k = k_walk<E, QUAD, PAIRS>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWalkSmem);
  int b = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k, kWalkThreads, kWalkSmem);
  return b > 0 ? b : 1;
}

template <class E, bool QUAD>
static int occ() {
  return std::min(occ_of<E, QUAD, true>(), occ_of<E, QUAD, false>());
}

static int walk_blocks_per_sm_query(int precision, bool quad, bool mask) {
  if (precision == 0) {
    if (mask) return walk_unsoftened_blocks_per_sm(quad);
    return quad ? occ<SplitEval<true>, true>() : occ<SplitEval<false>, false>();
  }
  if (quad) return mask ? occ<F64Eval<true, true>, true>() : occ<F64Eval<true, false>, true>();
  return mask ? occ<F64Eval<false, true>, false>() : occ<F64Eval<false, false>, false>();
}

// Cached: queried (and the kernels' shared-memory limit raised) once per
// variant, before any stream capture uses it.
int walk_blocks_per_sm(int precision, bool quad, bool mask) {
  static int cache[2][2][2] = {};
  int& v = cache[precision != 0][quad][mask];
  if (v == 0) v = walk_blocks_per_sm_query(precision, quad, mask);
  return v;
}

int walk_threads() { return kWalkThreads; }

// Device bytes of one list slot: the partial list, and for the two-pass
// schedule the group's FP64 sums, list lengths, progress and partial lengths;
// and of a dense list.
size_t walk_slot_bytes() { return kListCap * sizeof(uint2) + kGroupMax * 3 * sizeof(double) + 3 * sizeof(uint32_t); }
size_t walk_dense_bytes() { return kDenseCap * sizeof(uint2); }

// Lays the slots out over `base`: the lists, sums, lengths and progress words
// (from a.gnl on 2 * slots words, kWalkPending before every walk), partial
// lengths, dense lists.
void walk_scratch(WalkArgs& a, void* base, size_t slots) {
  a.nslots = (uint32_t)slots;
  a.wlist = static_cast<uint2*>(base);
  a.gsum = reinterpret_cast<double*>(a.wlist + slots * kListCap);
  a.gnl = reinterpret_cast<uint32_t*>(a.gsum + slots * kGroupMax * 3);
  a.prog = a.gnl + slots;
  a.plen = a.prog + slots;
  a.dlist = reinterpret_cast<uint2*>(a.plen + slots);
}

// ---------------------------------------------------------------------------
// Unfused integrate phase: kick_one / drift_one (integrate.h:15-16) with
// stored accelerations (G*a).

__global__ void k_integrate(Particle* __restrict__ p, const double* __restrict__ acc, uint32_t n, const SysDev* sys,
                            const SysParam* prm, int nsys) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = (uint32_t)nsys;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (sys[mid].begin <= i) lo = mid;
      else hi = mid;
    }
    const double kd = prm[lo].kick_dt, dd = prm[lo].drift_dt;
    Particle P = p[i];
    for (int d = 0; d < 3; ++d) P.vel[d] = __dadd_rn(P.vel[d], __dmul_rn(kd, acc[3 * (size_t)i + d]));
    if (dd != 0.0)
      for (int d = 0; d < 3; ++d) P.pos[d] = __dadd_rn(P.pos[d], __dmul_rn(dd, P.vel[d]));
    p[i] = P;
  }
}

void launch_integrate(Particle* p, const double* accel, uint32_t n, const SysDev* sys, const SysParam* prm, int nsys,
                      int sms, cudaStream_t s) {
  k_integrate<<<sms * 4, 256, 0, s>>>(p, accel, n, sys, prm, nsys);
}

__global__ void k_eval_done(DevState* st) {
  if (st->status == 0u) {
    st->evals_ok += 1u;
    st->pp_total += st->pp;
    st->pc_total += st->pc;
  }
}

void launch_eval_done(DevState* st, cudaStream_t s) { k_eval_done<<<1, 1, 0, s>>>(st); }

// ---------------------------------------------------------------------------
// FP64 direct sum on sample rows (brute_force.h:15-28): every other particle
// of the system, accel_from_source with zero second moment, times G.
//
// A block holds `rows` sample rows (a power of two up to kDirRows), two per
// thread in registers, and the threads beyond rows / 2 split each tile of
// sources staged in shared memory; the sources are split over gridDim.y so
// that any number of rows fills the GPU (about 8 blocks of 128 threads per
// SM), and the parts are added in order by k_direct_add.  Bound by the FP64
// pipe: 17 operations per pair, 5 of them the reciprocal square root.
// The call with 4,096 rows of 1,048,576 particles takes 6.6 ms (7.5 with a
// branch of its own for each row's reciprocal); with one row
// per 8 threads, 128 blocks, a division and a square root per pair and the
// particles repacked by the host 66.7 ms.

constexpr int kDirRows = 256;
constexpr int kDirThreads = 128;

// 1 / (x sqrt(x)): an approximate reciprocal square root (about 20 bits) and
// one step of Householder's third-order iteration, y (1 + e / 2 + 3 e^2 / 8)
// with e = 1 - x y^2, which triples its bits; for values far enough from the
// ends of the range (2^-600 .. 2^600), `ordinary`.  Others - zero, the smallest,
// the largest, NaN - take the plain quotient.
__device__ __forceinline__ bool ordinary(double x) {
  return (uint32_t)__double2hiint(x) - (423u << 20) <= (1200u << 20);
}
__device__ __forceinline__ double inv_r3(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  y = fma(y * e, fma(0.375, e, 0.5), y);
  return y * y * y;
}

__global__ void __launch_bounds__(kDirThreads, 8) k_direct(const Particle* __restrict__ p, uint32_t n,
                                                           const uint32_t* __restrict__ idx, uint32_t ns, uint32_t rows,
                                                           uint32_t chunk, double eps2, double G,
                                                           double* __restrict__ out) {
  __shared__ double4 src[kDirThreads];
  __shared__ double red[kDirThreads][6];
  const uint32_t pairs = (rows + 1) >> 1, nsub = kDirThreads / pairs;  // thread (sub, pair): rows 2 pair, 2 pair + 1
  const uint32_t pair = threadIdx.x % pairs, sub = threadIdx.x / pairs;
  const uint32_t r0 = blockIdx.x * rows + 2 * pair, r1 = r0 + 1;
  const bool live0 = r0 < ns, live1 = rows > 1 && r1 < ns;
  const uint32_t me0 = live0 ? idx[r0] : 0xffffffffu, me1 = live1 ? idx[r1] : 0xffffffffu;
  const Particle& q0 = p[live0 ? me0 : 0u];
  const Particle& q1 = p[live1 ? me1 : 0u];
  const double x0 = q0.pos[0], y0 = q0.pos[1], z0 = q0.pos[2], x1 = q1.pos[0], y1 = q1.pos[1], z1 = q1.pos[2];
  double a0x = 0, a0y = 0, a0z = 0, a1x = 0, a1y = 0, a1z = 0;
  const uint32_t begin = blockIdx.y * chunk, end = min(n, begin + chunk);
  for (uint32_t base = begin; base < end; base += kDirThreads) {
    __syncthreads();
    if (base + threadIdx.x < end) {
      const Particle& q = p[base + threadIdx.x];
      src[threadIdx.x] = make_double4(q.pos[0], q.pos[1], q.pos[2], q.mass);
    }
    __syncthreads();
    const uint32_t cnt = min((uint32_t)kDirThreads, end - base);
    for (uint32_t k = sub; k < cnt; k += nsub) {
      const double4 s = src[k];
      const double d0x = s.x - x0, d0y = s.y - y0, d0z = s.z - z0;
      const double d1x = s.x - x1, d1y = s.y - y1, d1z = s.z - z1;
      const double v0 = d0x * d0x + d0y * d0y + d0z * d0z + eps2, v1 = d1x * d1x + d1y * d1y + d1z * d1z + eps2;
      // one branch for both rows, so that their chains run side by side
      double c0, c1;
      if (ordinary(v0) && ordinary(v1)) c0 = inv_r3(v0), c1 = inv_r3(v1);
      else c0 = 1.0 / (v0 * sqrt(v0)), c1 = 1.0 / (v1 * sqrt(v1));
      c0 = base + k == me0 ? 0.0 : s.w * c0;  // not itself
      c1 = base + k == me1 ? 0.0 : s.w * c1;
      a0x += c0 * d0x, a0y += c0 * d0y, a0z += c0 * d0z;
      a1x += c1 * d1x, a1y += c1 * d1y, a1z += c1 * d1z;
    }
  }
  double* r = red[threadIdx.x];
  r[0] = a0x, r[1] = a0y, r[2] = a0z, r[3] = a1x, r[4] = a1y, r[5] = a1z;
  __syncthreads();
  // the subsets' sums, in order; a part of its own per split, scaled if it is the only one
  const double scale = gridDim.y == 1 ? G : 1.0;
  double* o = out + (size_t)blockIdx.y * ns * 3;
  for (uint32_t i = threadIdx.x; i < 6 * pairs; i += kDirThreads) {
    const uint32_t pr = i / 6, c = i - 6 * pr, row = blockIdx.x * rows + 2 * pr + c / 3;
    if (row >= ns || (rows == 1 && c >= 3)) continue;
    double v = 0.0;
    for (uint32_t t = 0; t < nsub; ++t) v += red[t * pairs + pr][c];
    o[(size_t)row * 3 + c % 3] = scale * v;
  }
}

__global__ void k_direct_add(const double* __restrict__ parts, uint32_t splits, uint32_t m, double G,
                             double* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  double v = 0.0;
  for (uint32_t s = 0; s < splits; ++s) v += parts[(size_t)s * m + i];
  out[i] = G * v;
}

DirectPlan direct_plan(uint32_t n, uint32_t ns, int sms) {
  DirectPlan d;
  d.rows = 1;
  while (d.rows < (uint32_t)kDirRows && d.rows < ns) d.rows *= 2;
  d.blocks = (ns + d.rows - 1) / d.rows;
  // splits of at least four tiles
  const uint32_t want = ((uint32_t)sms * 8u + d.blocks - 1) / d.blocks, most = (n + 4 * kDirThreads - 1) / (4 * kDirThreads);
  const uint32_t splits = want < 1u ? 1u : want < most ? want : most;
  d.chunk = ((n + splits - 1) / splits + kDirThreads - 1) / kDirThreads * kDirThreads;
  d.splits = (n + d.chunk - 1) / d.chunk;
  return d;
}

void launch_direct(const Particle* p, uint32_t n, const uint32_t* idx, uint32_t ns, double eps2, double G,
                   const DirectPlan& d, double* parts, double* out, cudaStream_t s) {
  k_direct<<<dim3(d.blocks, d.splits), kDirThreads, 0, s>>>(p, n, idx, ns, d.rows, d.chunk, eps2, G,
                                                           d.splits > 1 ? parts : out);
  if (d.splits > 1) k_direct_add<<<(3 * ns + 127) / 128, 128, 0, s>>>(parts, d.splits, 3 * ns, G, out);
}

// ---------------------------------------------------------------------------
// Energies (integrate.h:27-43): kinetic, and the unsoftened pairwise
// potential over i < j.  Per-block partial sums in out2[2 * block + {0,1}].

constexpr int kEnThreads = 256;

__global__ void __launch_bounds__(kEnThreads) k_energy(const Particle* __restrict__ p, uint32_t begin, uint32_t n,
                                                       double G, double* __restrict__ out2) {
  __shared__ double4 src[kEnThreads];
  __shared__ double red[2][kEnThreads / 32];
  double ek = 0.0, ep = 0.0;
  const uint32_t i = blockIdx.x * kEnThreads + threadIdx.x;
  double4 t = make_double4(0, 0, 0, 0);
  if (i < n) {
    const Particle& P = p[begin + i];
    t = make_double4(P.pos[0], P.pos[1], P.pos[2], P.mass);
    ek = 0.5 * P.mass * (P.vel[0] * P.vel[0] + P.vel[1] * P.vel[1] + P.vel[2] * P.vel[2]);
  }
  for (uint32_t base = blockIdx.x * kEnThreads; base < n; base += kEnThreads) {
    __syncthreads();
    if (base + threadIdx.x < n) {
      const Particle& Q = p[begin + base + threadIdx.x];
      src[threadIdx.x] = make_double4(Q.pos[0], Q.pos[1], Q.pos[2], Q.mass);
    }
    __syncthreads();
    const uint32_t cnt = min((uint32_t)kEnThreads, n - base);
    if (i < n) {
      for (uint32_t k = 0; k < cnt; ++k) {
        if (base + k <= i) continue;
        const double4 s = src[k];
        const double dx = t.x - s.x, dy = t.y - s.y, dz = t.z - s.z;
        ep -= G * t.w * s.w / sqrt(dx * dx + dy * dy + dz * dz);
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    ek += __shfl_xor_sync(kFull, ek, o);
    ep += __shfl_xor_sync(kFull, ep, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = ek;
    red[1][threadIdx.x >> 5] = ep;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0, b = 0;
    for (int w = 0; w < kEnThreads / 32; ++w) a += red[0][w], b += red[1][w];
    out2[2 * blockIdx.x] = a;
    out2[2 * blockIdx.x + 1] = b;
  }
}

// Returns this launch's own error (cudaLaunchKernel reports it directly, so
// an unrelated earlier error left on the thread is neither returned nor cleared).
cudaError_t launch_energy(const Particle* p, uint32_t begin, uint32_t n, double G, double* out2, int, cudaStream_t s) {
  void* args[] = {(void*)&p, (void*)&begin, (void*)&n, (void*)&G, (void*)&out2};
  return cudaLaunchKernel((const void*)k_energy, dim3((n + kEnThreads - 1) / kEnThreads), dim3(kEnThreads), args, 0, s);
}

// ---------------------------------------------------------------------------
// FP32 FMA throughput calibration: 8 independent FMA chains per thread.

__global__ void k_fma_peak(float* out, int iters, float seed) {
  float r[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) r[k] = seed + threadIdx.x * 1e-7f + k;
  const float m = 0.9999999f, c = 1e-7f;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) r[k] = fmaf(r[k], m, c);
  }
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += r[k];
  if (s == 1234.5678f) out[blockIdx.x] = s;  // never true; keeps the chains live
}

double measure_fp32_peak(int device) {
  cudaSetDevice(device);
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  float* out = nullptr;
  cudaMalloc(&out, sizeof(float) * sms * 64);
  const int blocks = sms * 8, threads = 256, iters = 1 << 14;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  k_fma_peak<<<blocks, threads>>>(out, 256, 1.0f);
  cudaEventRecord(e0);
  for (int r = 0; r < 5; ++r) k_fma_peak<<<blocks, threads>>>(out, iters, 1.0f + r);
  cudaEventRecord(e1);
  cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  const double flops = 5.0 * blocks * threads * 8.0 * iters * 2.0;
  return ms > 0 ? flops / (ms * 1e-3) / 1e12 : 0.0;
}

}  // namespace bhg
