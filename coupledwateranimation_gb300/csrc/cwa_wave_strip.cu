// cwa_wave_strip.cu — the default form of the wave advance: K leapfrog steps
// per launch on warp-wide strips held in registers.
//
// The job is the stand-alone wave module's (the reference's
// StencilImage2DTripleBuffered driving wave_comp.glsl EvolveWave, :171-206, one
// dispatch per step).  A warp owns a strip of 128 columns (four neighbouring
// columns a lane) and marches up its rows.  With each new row y of u^n it
// computes row y - 1 of u^(n+1), row y - 2 of u^(n+2), ... and stores row
// y - K of u^(n+K) and u^(n+K-1).  A level needs the two newest rows of the
// level before it and the row just formed, so the whole pipeline is 8 K floats
// a lane; west and east neighbours are in the lane's own four columns or one
// shuffle away.  No barriers between warps, and shared memory only for the rows
// that come in: the box forms
// (cwa_wave_tma.cu) move 3 to 5 shared-memory words a cell-step, which bound
// them.  Of the 128 columns, the outer K (rounded up to whole float4s) on each
// side are halo, except at the domain's borders (with a halo there too, 230 x
// 3001 took three strips for two), and a strip's march starts K rows below its
// first output row.
// What bounds it is the float pipe (63% busy at 4096^2) and the operations'
// latency, at 8.3 us a step there with three sims interleaved (11.6 alone);
// the 128 x 32 boxes took 14.7 (17.1), the memory traffic of 8-step launches
// would take 5.7.  With plain register loads in place of the cp.async ring a
// step took 17.4 us alone, and with scalar operations, all borders by selects,
// 18.3.  Programmatic dependent launches made it 15.8: CTAs that wait hold
// the places of those that run.
//
// Each cell runs the single-step kernel's operations in the same order with
// the same clamped (Neumann) neighbours, so a launch equals K single wave
// passes bit for bit.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "cwa_internal.h"

namespace cwa {
namespace {

constexpr int kStripThreads = 128;
constexpr int C = 4;           // columns a lane
constexpr int kStripW = 32 * C;  // columns a warp holds

// Columns of halo on each side of a strip: K, in whole vectors.
__host__ __device__ constexpr int halo_x(int k) { return (k + 3) & ~3; }

__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }

// Two neighbouring columns in one 64-bit register pair: the packed float
// instructions round each half like the scalar ones and take half the issue
// slots.
typedef unsigned long long F2;
__device__ __forceinline__ F2 pack(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float lo(F2 v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return a;
}
__device__ __forceinline__ float hi(F2 v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return b;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// a * b, as a * b + (-0) with the -0 from memory: the assembler contracts
// packed multiplies and adds into fused ones whatever their rounding modifier
// says, and a launch has to round like the single passes do.
__device__ __forceinline__ F2 mul2(F2 a, F2 b, F2 neg_zero) {
  return fma2(a, b, neg_zero);
}

// What a strip's cells may meet: nothing but cells of the domain; the domain's
// borders, its last column last in its lane; the borders with the last column
// anywhere; those and the line source's column.
enum Meets { kInside = 0, kBorder = 1, kRagged = 2, kSource = 3 };

struct StripCtx {
  int W, H, gx;  // field size, this lane's first column
  F2 wa, neg_wb, lam, last_mul, last_add, neg_zero;
  F2 zero_deposit;
  int from, to;    // the strip's own columns: the ones it stores
  bool two_step;   // zero_deposit is added after the last product, not with it
  bool first_col;  // column gx is the domain's first
  int last;        // column gx + last is the domain's last; else C
  int source;      // column gx + source is the line source's; else C
};

// One new row of a level: n, m, s = the rows above, at and below of the level
// before, p = the row two levels before.
template <int MEETS>
__device__ __forceinline__ void strip_row(const StripCtx& c, const F2 (&n)[C / 2], const F2 (&m)[C / 2],
                                          const F2 (&s)[C / 2], const F2 (&p)[C / 2], F2 (&out)[C / 2]) {
  float v[C + 2];  // the row with its neighbours: v[1 + k] = column k
#pragma unroll
  for (int h = 0; h < C / 2; ++h) {
    v[1 + 2 * h] = lo(m[h]);
    v[2 + 2 * h] = hi(m[h]);
  }
  v[0] = __shfl_up_sync(0xffffffffu, v[C], 1);
  v[C + 1] = __shfl_down_sync(0xffffffffu, v[1], 1);
  if (MEETS != kInside && c.first_col) v[0] = v[1];
#pragma unroll
  for (int h = 0; h < C / 2; ++h) {
    float ew[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int k = 2 * h + q;
      float e = v[2 + k];
      if ((MEETS >= kRagged || (MEETS == kBorder && k == C - 1)) && c.last == k) e = v[1 + k];
      ew[q] = fadd(e, v[k]);
    }
    const F2 nb = add2(add2(n[h], s[h]), pack(ew[0], ew[1]));
    F2 u = add2(mul2(c.wa, m[h], c.neg_zero), mul2(c.lam, nb, c.neg_zero));
    u = add2(u, mul2(c.neg_wb, p[h], c.neg_zero));  // u - wb p
    u = fma2(c.last_mul, u, c.last_add);
    if (MEETS == kSource) {
      float a = lo(u), b = hi(u);
      if (c.source == 2 * h && a > 0.0001f) a = fadd(a, 0.001f);
      if (c.source == 2 * h + 1 && b > 0.0001f) b = fadd(b, 0.001f);
      u = pack(a, b);
    }
    if (c.two_step) u = add2(u, c.zero_deposit);
    out[h] = u;
  }
}

// One march step: row y of u^n (n) and row y - 1 of u^(n-1) (p) come in.
// A[j] / B[j]: the newest and the second newest row of level j; the new row of
// level j replaces B[j], so the callers swap A and B from row to row.  Leaves
// row y - K of u^(n+K) in n; A[K - 1] then holds that row of u^(n+K-1).
// Borders: the row past the domain's last is a copy of the last, and the row
// below the first a copy of the first, so each level sees its clamped
// neighbour.
template <int K, int MEETS>
__device__ __forceinline__ void strip_step(const StripCtx& c, int y, F2 (&n)[C / 2], F2 (&p)[C / 2],
                                           F2 (&A)[K][C / 2], F2 (&B)[K][C / 2]) {
#pragma unroll
  for (int j = 0; j < K; ++j) {
    if (MEETS != kInside && y - j >= c.H) {
#pragma unroll
      for (int h = 0; h < C / 2; ++h) n[h] = A[j][h];
    }
    F2 out[C / 2];
    strip_row<MEETS>(c, n, A[j], B[j], p, out);
#pragma unroll
    for (int h = 0; h < C / 2; ++h) {
      p[h] = B[j][h];
      B[j][h] = n[h];
    }
    if (MEETS != kInside && y - j == 0) {
#pragma unroll
      for (int h = 0; h < C / 2; ++h) A[j][h] = n[h];
    }
#pragma unroll
    for (int h = 0; h < C / 2; ++h) n[h] = out[h];
  }
}

// The rows ahead come in through a ring of shared memory that each lane fills
// and reads for itself (cp.async): the rows in flight cost no registers and
// no barrier, and a row's DRAM latency (about two rows' steps) is covered.
constexpr int kAhead = 4;

// 128 columns of row y of u^n and of row y - 1 of u^(n-1); without VEC also the
// four floats more that 128 columns off a 16-byte boundary reach into.
template <bool VEC>
struct StripRing {
  float u[kAhead][kStripW + (VEC ? 0 : C)];
  float p[kAhead][kStripW + (VEC ? 0 : C)];
};

// 16 bytes; zero fill, with src not read, where it is not inside.
__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool inside) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(inside ? 16 : 0) : "memory");
}

// A lane's columns of a row on a 16-byte boundary, zeros outside the domain.
__device__ __forceinline__ void strip_fetch(const StripCtx& c, const float* row, const float* field, bool row_in,
                                            float* dst) {
  const bool in = row_in && c.gx >= 0 && c.gx < c.W;
  cp_async16(dst, in ? row : field, in);
}

// The strip's columns of any row, from index at of the field on: the aligned
// words that cover it, 33 of them, as far as they start inside the field
// (fields are padded to 128 bytes).  Columns outside the domain hold whatever
// lies there, which no cell of the domain uses.
__device__ __forceinline__ void strip_fetch_any(const StripCtx& c, const float* field, int at, bool row_in, int lane,
                                                float* dst) {
  const int first = (at & ~(C - 1)) + C * lane, last = (at & ~(C - 1)) + kStripW, cells = c.W * c.H;
  bool in = row_in && first < cells;
  cp_async16(dst + C * lane, in ? field + first : field, in);
  if (lane == 0) {
    in = row_in && last < cells;
    cp_async16(dst + kStripW, in ? field + last : field, in);
  }
}

__device__ __forceinline__ void strip_read(const float* src, F2 (&v)[C / 2]) {
  const float4 q = *reinterpret_cast<const float4*>(src);
  v[0] = pack(q.x, q.y);
  v[1] = pack(q.z, q.w);
}

// C columns from off columns behind src on: two whole words and a choice that
// is the warp's (four single loads of lanes C apart would conflict four ways).
__device__ __forceinline__ void strip_read_any(const float* src, int off, F2 (&v)[C / 2]) {
  const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + C);
  float q[C] = {a.x, a.y, a.z, a.w};
  if (off & 2) {
    q[0] = a.z, q[1] = a.w, q[2] = b.x, q[3] = b.y;
    if (off & 1) q[0] = a.w, q[1] = b.x, q[2] = b.y, q[3] = b.z;
  } else if (off & 1) {
    q[0] = a.y, q[1] = a.z, q[2] = a.w, q[3] = b.x;
  }
  v[0] = pack(q[0], q[1]);
  v[1] = pack(q[2], q[3]);
}

template <bool VEC>
__device__ __forceinline__ void strip_store(const StripCtx& c, float* __restrict__ row, const F2 (&v)[C / 2]) {
  if (VEC) {
    *reinterpret_cast<float4*>(row) = make_float4(lo(v[0]), hi(v[0]), lo(v[1]), hi(v[1]));
  } else {
#pragma unroll
    for (int k = 0; k < C; ++k)
      if (c.gx + k >= c.from && c.gx + k < c.to) row[k] = k & 1 ? hi(v[k / 2]) : lo(v[k / 2]);
  }
}

template <int K, bool VEC, int MEETS>
__device__ __forceinline__ void strip_march(const StripCtx& c, const float* __restrict__ cur,
                                            const float* __restrict__ prev, float* __restrict__ out_cur,
                                            float* __restrict__ out_prev, int row0, int row1, bool stores,
                                            StripRing<VEC>& ring) {
  F2 A[K][C / 2], B[K][C / 2];
#pragma unroll
  for (int j = 0; j < K; ++j)
#pragma unroll
    for (int h = 0; h < C / 2; ++h) A[j][h] = B[j][h] = 0ull;
  const int lane = threadIdx.x & 31;
  const int y0 = max(row0 - K, 0), y1 = row1 + K;  // rows that come in: [y0, y1)
  const int x0 = c.gx - C * lane;
  // the next row to fetch: yf of u^n, yf - 1 of u^(n-1)
  int yf = y0;
  const float* fu = cur + ((long)yf * c.W + c.gx);
  const float* fp = prev + ((long)(yf - 1) * c.W + c.gx);
  auto fetch = [&]() {
    const int slot = (yf - y0) & (kAhead - 1);
    const bool u_in = yf < c.H, p_in = yf > y0 && yf <= c.H;
    if (VEC) {
      strip_fetch(c, fu, cur, u_in, ring.u[slot] + C * lane);
      strip_fetch(c, fp, prev, p_in, ring.p[slot] + C * lane);
      fu += c.W;
      fp += c.W;
    } else {
      const int at = yf * c.W + x0;
      strip_fetch_any(c, cur, at, u_in, lane, ring.u[slot]);
      strip_fetch_any(c, prev, at - c.W, p_in, lane, ring.p[slot]);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    ++yf;
  };
#pragma unroll 1
  for (int q = 0; q < kAhead - 1; ++q) fetch();
  float* so = out_cur + ((long)(y0 - K) * c.W + c.gx);  // row y - K at this lane's columns
  float* sp = out_prev + ((long)(y0 - K) * c.W + c.gx);
  // one row: fetch the row kAhead - 1 further (into the slot read last), wait
  // for this one
  auto row = [&](int y, F2(&up)[K][C / 2], F2(&old)[K][C / 2]) {
    if (!VEC) __syncwarp();  // every lane has read the slot
    fetch();
    asm volatile("cp.async.wait_group %0;" ::"n"(kAhead - 1) : "memory");
    if (!VEC) __syncwarp();  // every lane's words are there
    const int slot = (y - y0) & (kAhead - 1);
    F2 n[C / 2], p[C / 2];
    if (VEC) {
      strip_read(ring.u[slot] + C * lane, n);
      strip_read(ring.p[slot] + C * lane, p);
    } else {
      const int at = y * c.W + x0;
      strip_read_any(ring.u[slot] + C * lane, at & (C - 1), n);
      strip_read_any(ring.p[slot] + C * lane, (at - c.W) & (C - 1), p);
    }
    strip_step<K, MEETS>(c, y, n, p, up, old);
    if (stores && y - K >= row0 && y - K < row1) {
      strip_store<VEC>(c, so, n);
      strip_store<VEC>(c, sp, up[K - 1]);
    }
    so += c.W;
    sp += c.W;
  };
#pragma unroll 1
  for (int y = y0; y < y1; y += 2) {
    row(y, A, B);
    row(y + 1, B, A);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// VEC: every scene's width is a multiple of four.
template <int K, bool VEC>
__global__ void __launch_bounds__(kStripThreads, K > 4 ? 3 : 4)
    k_wave_strip(WaveStripArgs a, int32_t n_strips) {
  constexpr int kHalo = halo_x(K), kOwn = kStripW - 2 * kHalo;
  __shared__ __align__(128) StripRing<VEC> rings[kStripThreads / 32];
  const int i = blockIdx.x * (kStripThreads / 32) + (threadIdx.x >> 5);
  if (i >= n_strips) return;
  StripRing<VEC>& ring = rings[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const WaveStrip t = a.strips[i];
  const SceneDev* S = a.scenes + t.scene;
  // The last strip, unless it is also the first, starts up to three columns
  // early, so that the domain's last column is last in its lane.
  const int begin = t.sx * kOwn;
  const bool first = t.sx == 0, last = begin + kStripW >= S->nx;
  const int x0 = last && !first ? begin - ((C - (S->nx & (C - 1))) & (C - 1)) : begin;
  StripCtx c;
  c.W = S->nx;
  c.H = S->nz;
  c.gx = x0 + C * lane;
  c.wa = pack(S->wa, S->wa);
  c.neg_wb = pack(-S->wb, -S->wb);
  c.lam = pack(S->lam, S->lam);
  c.neg_zero = pack(a.neg_zero, a.neg_zero);
  // The step ends with atten * u, then (coupled) + gain * (0 deposits).  With
  // one of the two missing or atten = 1 that is one fused operation with the
  // same rounding: 1 * u + zd, or atten * u + (-0).  The line source's test
  // lies between the two, so its strips keep them apart.
  const int src = c.W / 2;
  const bool source = S->line_source && src >= x0 && src < x0 + kStripW;
  const float zd = S->coupled ? fmul(S->gain, fmul(0.0f, S->dq)) : 0.0f;
  const bool fused = S->coupled && S->atten == 1.0f && !source;
  c.last_mul = pack(S->atten, S->atten);
  c.last_add = fused ? pack(zd, zd) : c.neg_zero;
  c.two_step = S->coupled && !fused;
  c.zero_deposit = pack(zd, zd);
  c.first_col = c.gx == 0;
  c.last = c.W - 1 >= c.gx && c.W - 1 < c.gx + C ? c.W - 1 - c.gx : C;
  c.from = first ? 0 : begin + kHalo;
  c.to = last ? c.W : begin + kHalo + kOwn;
  c.source = S->line_source && src >= c.gx && src < c.gx + C ? src - c.gx : C;
  const bool stores = c.gx + C > c.from && c.gx < c.to;
  const bool border = first || last || t.row0 - K < 0 || t.row1 + K > c.H;
  const float *cur = a.in_cur + S->woff, *prev = a.in_prev + S->woff;
  float *oc = a.out_cur + S->woff, *op = a.out_prev + S->woff;
  if (source)
    strip_march<K, VEC, kSource>(c, cur, prev, oc, op, t.row0, t.row1, stores, ring);
  else if (!VEC && first && last)
    strip_march<K, VEC, kRagged>(c, cur, prev, oc, op, t.row0, t.row1, stores, ring);
  else if (border)
    strip_march<K, VEC, kBorder>(c, cur, prev, oc, op, t.row0, t.row1, stores, ring);
  else
    strip_march<K, VEC, kInside>(c, cur, prev, oc, op, t.row0, t.row1, stores, ring);
}

}  // namespace

// Strips of about two resident CTAs a SM: a warp's step is a chain of dependent
// float operations, so two to three warps a scheduler run side by side, and
// longer strips recompute less (a strip of R rows marches R + 2 K).  Measured
// at K 8 (us a step; one sim, and per step with three sims interleaved): 4096^2
// in one / two / three CTAs a SM 13.7 / 11.6 / 11.5 and 9.6 / 8.3 / 8.9; 2048^2
// 4.4 / 4.2 / 4.6 and 3.0 / 2.9 / 3.5.  Where two CTAs a SM would cut strips
// below 32 rows, one CTA a SM: 4 / 5 / 8 warps a SM took 1400^2 2.8 / 3.6 / 3.1
// and 1.79 / 1.75 / 1.84, 4064 x 404 at K 6 2.7 / 3.4 / 3.1 and 1.55 / 1.55 /
// 1.58.  At least kWaveStripMinRows rows: 773 x 1021 with 8 /
// 16 / 32 rows 3.3 / 3.1 / 4.1 and 1.8 / 1.6 / 1.7.
void wave_strips(const std::vector<SceneDev>& scenes, int steps, int sms, std::vector<WaveStrip>* out) {
  const int halo = halo_x(steps), w = kStripW - 2 * halo;
  double area = 0.0;
  for (const SceneDev& d : scenes) area += (double)d.nx * d.nz;
  for (size_t s = 0; s < scenes.size(); ++s) {
    const SceneDev& d = scenes[s];
    const int nsx = std::max(1, (d.nx - 2 * halo + w - 1) / w);
    auto segments = [&](double warps_per_sm) {
      return (int)(warps_per_sm * sms * ((double)d.nx * d.nz / area) / nsx);
    };
    int nsy = segments(8.0);
    if (nsy > d.nz / 32) nsy = std::max(d.nz / 32, segments(4.0));
    nsy = std::max(1, std::min(nsy, d.nz / kWaveStripMinRows));
    for (int q = 0; q < nsy; ++q) {
      const int r0 = (int)((int64_t)d.nz * q / nsy), r1 = (int)((int64_t)d.nz * (q + 1) / nsy);
      for (int x = 0; x < nsx; ++x) out->push_back(WaveStrip{(int32_t)s, x, r0, r1});
    }
  }
}

cudaError_t launch_wave_strips(const WaveStripArgs& a, int32_t n_strips, int steps, cudaStream_t stream) {
  if (n_strips <= 0) return cudaSuccess;
  const int per = kStripThreads / 32, grid = (n_strips + per - 1) / per;
  switch (steps) {
#define CWA_STRIP(K) \
  case K:                                                                     \
    if (a.whole)                                                              \
      k_wave_strip<K, true><<<grid, kStripThreads, 0, stream>>>(a, n_strips); \
    else                                                                      \
      k_wave_strip<K, false><<<grid, kStripThreads, 0, stream>>>(a, n_strips); \
    break
    CWA_STRIP(4);
    CWA_STRIP(5);
    CWA_STRIP(6);
    CWA_STRIP(7);
    CWA_STRIP(8);
#undef CWA_STRIP
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace cwa
