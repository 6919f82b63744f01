// cwa_device.cuh — device helpers shared by the kernels: the float32 cell
// hash and the bilinear height-field sample, both written one rounding per
// operation (__f*_rn) so results do not depend on FMA contraction.
#pragma once

#include <cuda_runtime.h>

#include "cwa_internal.h"

namespace cwa {

// clamp(floor((p - lo) / cell), 0, n - 1)  (UniformGrid2D/ugrid_particles_cs.glsl:97-103)
__device__ __forceinline__ int cell_axis(float p, float lo, float cell, int n) {
  float t = __fdiv_rn(__fsub_rn(p, lo), cell);
  float f = floorf(t);
  f = fminf(fmaxf(f, 0.0f), (float)(n - 1));
  return (int)f;
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Programmatic dependent launch across a step's kernel chain.  Every kernel
// of the chain first waits for the kernel before it to complete (a no-op
// when it was launched without the chaining attribute), then lets the next
// kernel be launched, whose blocks take the SMs this grid's last wave frees
// and wait there: launch latency and ramp-up overlap this grid's tail.  The
// wait covers every earlier kernel, since each one waited for its own
// predecessor before it could complete.
__device__ __forceinline__ void chain_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Index checks of the debug build (compiled with CWA_DEBUG_CHECKS): a failed
// check records kStatusBounds in the status word and evaluates to true, so
// the caller skips the access; release builds compile every check to false.
// They stand in for a memory checker: no trap, the context stays usable.
__device__ __forceinline__ bool dcheck_failed(bool ok, int32_t* status) {
  if (!ok && status) atomicOr(status, kStatusBounds);
  return !ok;
}
#ifdef CWA_DEBUG_CHECKS
#define CWA_DCHECK_FAILED(cond, status) (::cwa::dcheck_failed((cond), (status)))
#else
#define CWA_DCHECK_FAILED(cond, status) (false)
#endif

__device__ __forceinline__ bool finite3(float4 p) {
  return isfinite(p.x) && isfinite(p.y) && isfinite(p.z);
}

// Warp-aggregated count: the lanes of a warp with the same key share one
// atomicAdd; each lane's slot is its arrival rank within the cell.  The lanes
// are grouped by five bits of a multiplicative hash of the key, a ballot a bit;
// of a group the lanes that hold its first lane's key go together, of the rest
// those that hold the rest's first key, any others (three keys of one hash
// among 32 lanes) each alone.
// Point grid builds of 1,000,003 points, us, with the atomics of runs of equal
// neighbours joined / of all equal keys by match.any / by this:
//   scattered over 8,192 cells              58 /  66 /  58
//   sorted, all in one cell                 46 /  46 /  46
//   two cells in turn                      360 /  46 /  46
//   every other one in one cell, the rest scattered over 400,000
//                                          355 /  54 /  52
// match.any takes a step for each distinct key of the warp; runs leave equal
// keys with others between them to the memory system, one by one.
__device__ __forceinline__ int count_slot(int32_t* count, int key) {
  const unsigned int active = __activemask();
  const int lane = threadIdx.x & 31;
  const unsigned int hash = ((unsigned int)key * 0x9e3779b1u) >> 27;
  unsigned int peers = active;
#pragma unroll
  for (int b = 0; b < 5; ++b) {
    const bool bit = (hash >> b) & 1u;
    const unsigned int set = __ballot_sync(active, bit);
    peers &= bit ? set : ~set;
  }
#pragma unroll
  for (int round = 0; round < 2; ++round) {
    const bool same = __shfl_sync(active, key, __ffs((int)peers) - 1) == key;
    const unsigned int all = __ballot_sync(active, same);
    peers &= same ? all : round == 0 ? ~all : 1u << lane;
  }
  const int leader = __ffs((int)peers) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(count + key, __popc(peers));
  base = __shfl_sync(active, base, leader);
  return base + __popc(peers & ((1u << lane) - 1u));
}

// The same for particles that lie in cell order, or did a step ago: only runs
// of equal neighbours share an atomic, for a shuffle and a ballot (ten steps of
// 1M particles with count_slot in the integration take 0.2% longer).
__device__ __forceinline__ int count_slot_sorted(int32_t* count, int key) {
  const unsigned int active = __activemask();
  const int lane = threadIdx.x & 31;
  const int prev = __shfl_up_sync(active, key, 1);
  const bool first = lane == 0 || !((active >> (lane - 1)) & 1u) || prev != key;
  const unsigned int firsts = __ballot_sync(active, first);
  // the run: from the nearest first at or below this lane to the lane before
  // the next first or the next inactive lane
  const int begin = 31 - __clz(firsts & (0xffffffffu >> (31 - lane)));
  int base = 0;
  if (first) {
    const unsigned int stop = (firsts | ~active) & ~(0xffffffffu >> (31 - lane));  // lanes above this one
    const int end = stop ? __ffs(stop) - 1 : 32;
    base = atomicAdd(count + key, end - lane);
  }
  base = __shfl_sync(active, base, begin);
  return base + lane - begin;
}

// texture(wave_tex, uv) with GL_LINEAR / GL_CLAMP_TO_EDGE on an R32F image
// (StencilImage2DTripleBuffered.cpp:21-26): texel centres at (i + 0.5) / W.
struct Bilinear {
  float v00, v10, v01, v11, ax, ay;
};

__device__ __forceinline__ Bilinear bilinear_patch(const float* __restrict__ u, int w, int h, float s,
                                                   float t) {
  float tx = __fsub_rn(__fmul_rn(s, (float)w), 0.5f);
  float ty = __fsub_rn(__fmul_rn(t, (float)h), 0.5f);
  tx = fminf(fmaxf(tx, -1.0f), (float)w);
  ty = fminf(fmaxf(ty, -1.0f), (float)h);
  float fx = floorf(tx), fy = floorf(ty);
  Bilinear b;
  b.ax = __fsub_rn(tx, fx);
  b.ay = __fsub_rn(ty, fy);
  int x0 = (int)fx, y0 = (int)fy;
  int x1 = clampi(x0 + 1, 0, w - 1), y1 = clampi(y0 + 1, 0, h - 1);
  x0 = clampi(x0, 0, w - 1);
  y0 = clampi(y0, 0, h - 1);
  b.v00 = __ldg(u + (size_t)y0 * w + x0);
  b.v10 = __ldg(u + (size_t)y0 * w + x1);
  b.v01 = __ldg(u + (size_t)y1 * w + x0);
  b.v11 = __ldg(u + (size_t)y1 * w + x1);
  return b;
}

__device__ __forceinline__ float bilinear_value(const Bilinear& b, float* top_out = nullptr,
                                                float* bot_out = nullptr) {
  float bx = __fsub_rn(1.0f, b.ax);
  float top = __fadd_rn(__fmul_rn(bx, b.v00), __fmul_rn(b.ax, b.v10));
  float bot = __fadd_rn(__fmul_rn(bx, b.v01), __fmul_rn(b.ax, b.v11));
  if (top_out) *top_out = top;
  if (bot_out) *bot_out = bot;
  return __fadd_rn(__fmul_rn(__fsub_rn(1.0f, b.ay), top), __fmul_rn(b.ay, bot));
}

__device__ __forceinline__ float sample_height(const float* __restrict__ u, int w, int h, float s, float t) {
  return bilinear_value(bilinear_patch(u, w, h, s, t));
}

// Value and derivatives along the texel axes of the same bilinear patch.
__device__ __forceinline__ void sample_height_grad(const float* __restrict__ u, int w, int h, float s,
                                                   float t, float* val, float* dtx, float* dty) {
  Bilinear b = bilinear_patch(u, w, h, s, t);
  float top, bot;
  float by = __fsub_rn(1.0f, b.ay);
  *val = bilinear_value(b, &top, &bot);
  *dtx = __fadd_rn(__fmul_rn(by, __fsub_rn(b.v10, b.v00)), __fmul_rn(b.ay, __fsub_rn(b.v11, b.v01)));
  *dty = __fsub_rn(bot, top);
}

}  // namespace cwa
