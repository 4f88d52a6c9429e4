// Device helpers shared by the walk kernels (bhg_walk.cu, bhg_walk_unsoftened.cu).
#pragma once

#include "bhg_kernels.h"

namespace bhg {

constexpr uint32_t kFull = 0xffffffffu;
constexpr float kFarAway = 1.0e10f;  // padding source: contributes exactly 0
constexpr int kWalkWarps = 4;
constexpr int kWalkThreads = kWalkWarps * 32;
constexpr uint32_t kListCap = 4096;  // entries of a list of the sources some targets of a group take (32 KB)
// a group's list length(s) before its shared walk has finished (two-pass
// schedule; set before every walk)
constexpr uint32_t kListPending = kWalkPending;
// ... and when the job that was to publish it gave up waiting itself
constexpr uint32_t kListLost = 0xfffffffeu;

__device__ __forceinline__ uint32_t warp_incl_scan_u32(uint32_t v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t u = __shfl_up_sync(kFull, v, o);
    if (lane >= o) v += u;
  }
  return v;
}

// Squared distance from (x, y, z) to the nearest point of the box, as
// BBox::near2 (multipole.h:132-136) rounds it.
__device__ __forceinline__ double near2(const double lo[3], const double hi[3], double x, double y, double z) {
  double dx = fmax(fmax(__dsub_rn(lo[0], x), __dsub_rn(x, hi[0])), 0.0);
  double dy = fmax(fmax(__dsub_rn(lo[1], y), __dsub_rn(y, hi[1])), 0.0);
  double dz = fmax(fmax(__dsub_rn(lo[2], z), __dsub_rn(z, hi[2])), 0.0);
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// Squared distance to the farthest point of the box (BBox::far2, multipole.h:137-141).
__device__ __forceinline__ double far2(const double lo[3], const double hi[3], double x, double y, double z) {
  double dx = fmax(__dsub_rn(x, lo[0]), __dsub_rn(hi[0], x));
  double dy = fmax(__dsub_rn(y, lo[1]), __dsub_rn(hi[1], y));
  double dz = fmax(__dsub_rn(z, lo[2]), __dsub_rn(hi[2], z));
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// 32 bytes of device memory in one load (the SM's widest): a gather of
// records takes half the passes through the load unit that 16-byte loads take.
__device__ __forceinline__ void ld32(const void* p, double& a, double& b, double& c, double& d) {
  asm("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(a), "=d"(b), "=d"(c), "=d"(d)
      : "l"(__cvta_generic_to_global(p)));
}
__device__ __forceinline__ void ld32(const void* p, float (&v)[8]) {
  asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
      : "l"(__cvta_generic_to_global(p)));
}

// rsqrt.approx.ftz.f32 (PTX ISA): the approximate reciprocal square root,
// subnormal inputs and results flushed to zero.  The split evaluator's r^2 is
// in units scaled to the system's size (at least eps^2 there, or masked when
// eps = 0), so the flush only drops contributions below FP32's normal range.
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Bounding box of particles [b, b + T) (BBox::add, multipole.h:121-128).
__device__ __forceinline__ void particle_box(const double4* pm, uint32_t b, uint32_t T, int lane, double lo[3],
                                             double hi[3]) {
  lo[0] = lo[1] = lo[2] = INFINITY;
  hi[0] = hi[1] = hi[2] = -INFINITY;
  for (uint32_t i = lane; i < T; i += 32) {
    const double4 q = pm[b + i];
    lo[0] = fmin(lo[0], q.x), hi[0] = fmax(hi[0], q.x);
    lo[1] = fmin(lo[1], q.y), hi[1] = fmax(hi[1], q.y);
    lo[2] = fmin(lo[2], q.z), hi[2] = fmax(hi[2], q.z);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      lo[d] = fmin(lo[d], __shfl_xor_sync(kFull, lo[d], o));
      hi[d] = fmax(hi[d], __shfl_xor_sync(kFull, hi[d], o));
    }
  }
}

// on_result(particle, G * acc) (grouped_ttg.h:281-283), then kick_one /
// drift_one (integrate.h:15-16), for particles p0 .. p0 + n - 1 whose FP64
// sums are in sums[0 .. n).
__device__ __forceinline__ void kick_drift(const WalkArgs& a, const SysParam& sp, const double (*sums)[3], uint32_t p0,
                                           uint32_t n, int lane) {
  for (uint32_t i = lane; i < n; i += 32) {
    const uint32_t p = p0 + i;
    const double gx = __dmul_rn(sp.G, sums[i][0]), gy = __dmul_rn(sp.G, sums[i][1]), gz = __dmul_rn(sp.G, sums[i][2]);
    if (a.accel) {
      a.accel[3 * (size_t)p + 0] = gx;
      a.accel[3 * (size_t)p + 1] = gy;
      a.accel[3 * (size_t)p + 2] = gz;
    }
    Particle P = a.staged[p];
    P.vel[0] = __dadd_rn(P.vel[0], __dmul_rn(sp.kick_dt, gx));
    P.vel[1] = __dadd_rn(P.vel[1], __dmul_rn(sp.kick_dt, gy));
    P.vel[2] = __dadd_rn(P.vel[2], __dmul_rn(sp.kick_dt, gz));
    if (sp.drift_dt != 0.0) {
      P.pos[0] = __dadd_rn(P.pos[0], __dmul_rn(sp.drift_dt, P.vel[0]));
      P.pos[1] = __dadd_rn(P.pos[1], __dmul_rn(sp.drift_dt, P.vel[1]));
      P.pos[2] = __dadd_rn(P.pos[2], __dmul_rn(sp.drift_dt, P.vel[2]));
    }
    a.out[p] = P;
  }
  __syncwarp();
}

// The system holding particle p (systems lie back to back).
__device__ __forceinline__ uint32_t system_of(const WalkArgs& a, uint32_t p) {
  uint32_t lo = 0, hi = (uint32_t)a.nsys;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a.sys[mid].begin <= p) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Whether another launch walks system s.
__device__ __forceinline__ bool walked_elsewhere(const WalkArgs& a, uint32_t s) {
  return a.only != WalkOnly::kAll && (a.prm[s].eps2 > 0.0) != (a.only == WalkOnly::kSoftened);
}

// A target job's wait, by a warp, for its group's list length(s): them, or
// kListLost.  Bounded: after `limit` polls it sets kStSpinLimit, so that the
// kernel ends without the job and the host reports the error.
__device__ __forceinline__ uint32_t wait_lengths(const uint32_t* length, int limit, DevState* st, int lane) {
  uint32_t len = ld_volatile(length);
  for (int spins = 0; len == kListPending && spins < limit; ++spins) {
    __nanosleep(128);
    len = ld_volatile(length);
  }
  len = __shfl_sync(kFull, len, 0);  // one value for the warp
  if (len != kListPending) return len;
  if (lane == 0) atomicOr(&st->status, kStSpinLimit);
  return kListLost;
}

// The group of walk group gi: its targets, first particle and system.
struct GroupInfo {
  uint32_t t0, k, p0, s;
};

__device__ __forceinline__ GroupInfo group_info(const WalkArgs& a, uint32_t gi, uint32_t ngroups, uint32_t ntargets) {
  GroupInfo g;
  g.t0 = a.groups[gi];
  g.k = (gi + 1 < ngroups ? a.groups[gi + 1] : ntargets) - g.t0;
  g.p0 = a.nbegin[a.targets[g.t0]];
  g.s = a.nsys > 1 ? system_of(a, g.p0) : 0u;
  return g;
}

// The unsoftened split walk (bhg_walk_unsoftened.cu).
void launch_walk_unsoftened(const WalkArgs& a, bool quad, int grid, cudaStream_t s);
int walk_unsoftened_blocks_per_sm(bool quad);

}  // namespace bhg
