// cwa_sph.cu — SPH neighbour passes over the cell-sorted particle arrays.
//
//   rho_pres: poly6 density, equation of state, and (REFERENCE_3D) the wave
//             density / pressure terms — CoupledWaterAnimation/rho_pres_comp.glsl:49-81.
//   force:    spiky pressure gradient + viscosity Laplacian, then either the
//             reference's crest / torque / drag / wave-normal terms
//             (force_comp.glsl:62-139) or gravity only (MULLER).
//
// The reference loops over all N particles per particle (O(N^2)).  Here the
// particles are sorted by uniform-grid cell (x/y cell edge >= the search
// radius), so the candidates of a particle lie in 9 rows (columns x-1..x+1,
// y-1..y+1) of the sorted arrays, each a contiguous z range.  Every pair with
// r < h lies inside them, so the neighbour sets equal the shaders'.
//
// Two modes (cwa_sim_options.verlet_skin):
//  * per-step (skin 0): k_scan_cands tests every candidate of the particle's
//    rows once, accumulates the density and keeps the hits as this step's
//    neighbour list;
//  * Verlet (skin > 0): the grid and a list of every pair within
//    h (1 + skin) are rebuilt only when some particle has moved more than
//    skin h / 2 since the last rebuild (integrate raises a device flag);
//    k_rho_list walks that list each step, tests r < h and keeps the hits.
// Either way force runs its pair terms over the step's hits only.
//
// A row's cell-based start is start[row + max(cz - rz, 0)], decodable from
// the particle's sorted cell key alone.  The step's hits are nine 64-bit
// row masks per particle (bit b = the row's candidate at that start + b):
// the density pass sets bits in registers, with no per-hit store, and force
// walks the set bits.  The Verlet list holds 16-bit codes (row << 12 |
// offset from the same start), so it stays valid while the particles move.
// The candidate scan can stage the CTA's rows in shared memory with bulk
// TMA copies (cp.async.bulk, completion on an mbarrier).
//
// Sums are accumulated in one of three precisions (template P):
//   CWA_PREC_FP32 plain float; CWA_PREC_COMPENSATED float partial sums (per
//   row or per 8 pairs) folded into a Knuth two-sum accumulator;
//   CWA_PREC_FP64 double pair math and sums.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "cwa_device.cuh"
#include "cwa_internal.h"

namespace cwa {
namespace {

template <int P>
struct Sum {
  float s = 0.0f;
  __device__ __forceinline__ void add(float x) { s += x; }
  __device__ __forceinline__ float get() const { return s; }
};

template <>
struct Sum<CWA_PREC_COMPENSATED> {
  float s = 0.0f, c = 0.0f;
  __device__ __forceinline__ void add(float x) {
    float t = __fadd_rn(s, x);
    float bp = __fsub_rn(t, s);
    c = __fadd_rn(c, __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(x, bp)));
    s = t;
  }
  __device__ __forceinline__ float get() const { return s + c; }
};

template <>
struct Sum<CWA_PREC_FP64> {
  double s = 0.0;
  __device__ __forceinline__ void add(double x) { s += x; }
  __device__ __forceinline__ double get() const { return s; }
};

template <int P>
using Real = typename std::conditional<P == CWA_PREC_FP64, double, float>::type;

__device__ __forceinline__ float inv_sqrt(float x) { return rsqrtf(x); }
__device__ __forceinline__ double inv_sqrt(double x) { return rsqrt(x); }
__device__ __forceinline__ float recip(float x) { return __fdividef(1.0f, x); }
__device__ __forceinline__ double recip(double x) { return 1.0 / x; }

// (double)f without the conversion instruction.  GB300 runs every FP64
// instruction, float <-> double conversions included, at 2 lanes a clock and
// SM; the integer form runs at 64.  Zeros, denormals, infinities and NaNs
// take the instruction.
__device__ __forceinline__ double widen(float f) {
  const uint32_t u = __float_as_uint(f);
  if (((u >> 23) + 1u & 0xffu) <= 1u) return (double)f;
  return __hiloint2double((int)((u & 0x80000000u) | (((u >> 3) & 0x0fffffffu) + 0x38000000u)), (int)(u << 29));
}
__device__ __forceinline__ float widen_as(float f, float) { return f; }
__device__ __forceinline__ double widen_as(float f, double) { return widen(f); }

// a - b in the precision of the third argument's type, the operands being
// floats.  In double: the float difference is exact unless the operands
// differ by more than a factor of 2 (positions near a coordinate plane); its
// error (exact, Knuth's two-sum) is added back there, so the result equals
// the double difference of the operands, for one integer conversion instead
// of two conversions and a subtraction in FP64.
__device__ __forceinline__ float diff_as(float a, float b, float) { return a - b; }
__device__ __forceinline__ double diff_as(float a, float b, double) {
  const float d = __fsub_rn(a, b);
  const float bb = __fsub_rn(d, a);
  const float e = __fsub_rn(__fsub_rn(a, __fsub_rn(d, bb)), __fadd_rn(b, bb));
  double x = widen(d);
  if (fabsf(e) > 0.0f) x += widen(e);
  return x;
}

struct CellCoord {
  int x, y, z;
};

// Cell coordinates of a global cell id (the two divisions by the scene's
// grid dimensions as multiply-highs with the scene's exact magic numbers).
__device__ __forceinline__ CellCoord cell_of_key(const SceneDev* S, int key) {
  const int local = key - S->coff, nz = S->dims[2], ny = S->dims[1];
  const int xy = (int)(((unsigned long long)(uint32_t)local * S->mz) >> S->sz);
  CellCoord c;
  c.z = local - xy * nz;
  c.x = (int)(((unsigned long long)(uint32_t)xy * S->my) >> S->sy);
  c.y = xy - c.x * ny;
  return c;
}

__device__ __forceinline__ bool row_valid(const SceneDev* S, CellCoord c, int r) {
  const int x = c.x + r / 3 - 1, y = c.y + r % 3 - 1;
  return x >= 0 && x < S->dims[0] && y >= 0 && y < S->dims[1];
}

__device__ __forceinline__ int row_id(const SceneDev* S, CellCoord c, int r) {
  const int nz = S->dims[2], nyz = S->dims[1] * nz;
  return S->coff + c.x * nyz + c.y * nz + (r / 3 - 1) * nyz + (r % 3 - 1) * nz;
}

// Cell-based start of each row: the base that row-mask bits and Verlet codes are relative
// to.  rz z cells below the particle's cell cover every window.
__device__ __forceinline__ void row_bases(const SceneDev* S, const int32_t* __restrict__ start, CellCoord c,
                                          int base[9]) {
  const int z0 = max(c.z - S->rz, 0);
#pragma unroll
  for (int r = 0; r < 9; ++r) base[r] = row_valid(S, c, r) ? __ldg(start + row_id(S, c, r) + z0) : 0;
}

// Sorted-index ranges [b, e) of the candidates within radius sqrt(rad2) of
// p, row by row.  A row whose column is farther than the radius in (x, y)
// is empty; the others cover the z cells of the window
// |z - pz| < sqrt(rad2 - d^2), d = the column's (x, y) distance.  The
// radius carries a 2^-10 margin (about h / 1024 of slack in the window), so
// neither float rounding nor the approximate square root t * rsqrt(t)
// (relative error ~1e-7) ever drops a pair.
//
// An out-of-domain column is infinitely far, so one comparison rules out
// either kind of row.  Nine windows a particle are a fifth of the density
// pass's instructions, so each is kept short: one conversion that rounds down
// a bound, no scaling around the square root (ten steps of 1M particles,
// three sims interleaved, 3750 to 3585 us).
//
// Every kernel forms the same window from the same position, bit for bit: the
// masks of a dense spot count from the windows' starts, which the density pass
// and force form in different kernels.  So each operation names its rounding
// and none is left for the compiler to contract.
struct RowWindows {
  float dxm, dxp, dym, dyp, zl, izc, zmax, rad2;
  __device__ __forceinline__ RowWindows(const SceneDev* S, float4 p, CellCoord c, float r2) {
    const float x0f = __fmaf_rn((float)c.x, S->cell, S->lo[0]);
    const float y0f = __fmaf_rn((float)c.y, S->cell, S->lo[1]);
    const float far = __int_as_float(0x7f800000);
    dxm = c.x > 0 ? fmaxf(__fsub_rn(p.x, x0f), 0.0f) : far;
    dxp = c.x + 1 < S->dims[0] ? fmaxf(__fsub_rn(__fadd_rn(x0f, S->cell), p.x), 0.0f) : far;
    dym = c.y > 0 ? fmaxf(__fsub_rn(p.y, y0f), 0.0f) : far;
    dyp = c.y + 1 < S->dims[1] ? fmaxf(__fsub_rn(__fadd_rn(y0f, S->cell), p.y), 0.0f) : far;
    zl = __fsub_rn(p.z, S->lo[2]);
    izc = S->inv_cellz;
    zmax = (float)(S->dims[2] - 1);
    rad2 = r2;
  }
  // the z cell of height z over the grid's lowest, clamped to the grid
  __device__ __forceinline__ int zcell(float z) const {
    return __float2int_rd(fminf(fmaxf(__fmul_rn(z, izc), 0.0f), zmax));
  }
  __device__ __forceinline__ void range(const SceneDev* S, const int32_t* __restrict__ start, CellCoord c, int r,
                                        int& b, int& e) const {
    const int dx = r / 3 - 1, dy = r % 3 - 1;
    const float ddx = dx < 0 ? dxm : (dx > 0 ? dxp : 0.0f);
    const float ddy = dy < 0 ? dym : (dy > 0 ? dyp : 0.0f);
    const float d2 = __fmaf_rn(ddx, ddx, __fmul_rn(ddy, ddy));
    const bool ok = d2 < rad2;
    const float t = fmaxf(__fsub_rn(rad2, d2), 1e-30f);
    float w;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(w) : "f"(t));
    w = __fmul_rn(t, w);
    const int row = row_id(S, c, r);
    b = e = 0;
    if (ok) {
      b = __ldg(start + (row + zcell(__fsub_rn(zl, w))));
      e = __ldg(start + (row + zcell(__fadd_rn(zl, w)) + 1));
    }
  }
};

__device__ __forceinline__ void row_ranges(const SceneDev* S, const int32_t* __restrict__ start, float4 p,
                                           CellCoord c, float rad2, int b[9], int e[9]) {
  const RowWindows w(S, p, c, rad2);
#pragma unroll
  for (int r = 0; r < 9; ++r) w.range(S, start, c, r, b[r], e[r]);
}

__device__ __forceinline__ float uv_s(const SceneDev* S, float x) { return x * S->uvs[0] + S->uvo[0]; }
__device__ __forceinline__ float uv_t(const SceneDev* S, float z) { return z * S->uvs[1] + S->uvo[1]; }

// rho, p and the reference's wave terms (rho_pres_comp.glsl:70-80).
__device__ __forceinline__ float2 eos(const SceneDev* S, float rho, float4 pi, const float* __restrict__ wave) {
  float p = S->k * (rho - S->rho0);
  if (S->preset == CWA_PRESET_REFERENCE_3D) {
    p = fmaxf(p, 0.0f);
    const float H = sample_height(wave + S->woff, S->nx, S->nz, uv_s(S, pi.x), uv_t(S, pi.z));
    const float wf = H * rho;
    p += wf;
    rho += wf * S->inv_kr;
    rho = fmaxf(S->rho0, rho);
  }
  return make_float2(rho, p);
}

// Force's gather record of particle i: (x, y, z, p) and (vx, vy, vz, 1/rho)
// side by side, so a pair costs one aligned 32-byte gather (two of 16 bytes from
// two arrays: ten steps of 1M particles, three sims interleaved, 3010 us for
// 2868; four steps of 4.2M in FP32 5020 for 4740); 1/rho uses force's recip.
// FP64 keeps 1/rho in double beside them: one division a particle instead of
// one a pair.
__device__ __forceinline__ void load_pair(const PairRec* __restrict__ rec, float4& x, float4& v) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w), "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(rec));
}

template <int P>
__device__ __forceinline__ void write_pair_rec(PairRec* __restrict__ pairs, double* __restrict__ irho,
                                               const float4* __restrict__ vel, int i, float4 pi, float2 rp) {
  const float4 v = __ldg(vel + i);
  pairs[i].xp = make_float4(pi.x, pi.y, pi.z, rp.y);
  pairs[i].vr = make_float4(v.x, v.y, v.z, P == CWA_PREC_FP64 ? 0.0f : recip(rp.x));
  if (P == CWA_PREC_FP64) irho[i] = recip((double)rp.x);
}

// ---- shared-memory staging with bulk TMA copies --------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// One 128-bit shared load of a staged candidate at shared-window address a,
// so a quarter warp's eight lanes move 128 bytes per wavefront (the compiler
// would otherwise split the load when the fourth component is unused).  The
// row loop steps a 32-bit address: in place of converting a generic pointer
// at every candidate, that saves 113 instructions a warp and took the
// density pass from 154 to 147 us at 1M particles.
__device__ __forceinline__ float4 lds128(uint32_t a) {
  float4 v;
  asm("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// Global -> shared bulk copy (16-byte aligned addresses, size a multiple of 16).
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait on one phase of the staging barrier (phase parity 0 for a
// CTA's first stage, alternating in the work-queue form).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity = 0) {
  for (int k = 0; k < (1 << 20); ++k)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

constexpr int kNbThreads = 128;
constexpr int kStageCap = 1536;   // staged candidates per CTA (24 KB)
constexpr int kRowCodeBits = 12;  // a hit is (row << 12) | offset from the row's cell-based start
constexpr int kRowCodeMax = 1 << kRowCodeBits;
constexpr int kMaxCols = 3;       // columns a CTA's particles may span and still be staged
constexpr int kMaxSegs = 9 * kMaxCols;  // 27 row segments: one planning warp covers them

// Verlet lists hold codes in pairs: code k of particle i is half (k & 1) of
// the 32-bit word (k >> 1) * n + i, so a warp writes its lanes' k-th pairs as
// one 128-byte store and readers load two codes per load.
__device__ __forceinline__ uint32_t code_pair(const uint16_t* __restrict__ list, int k, int i, int n) {
  return __ldg(reinterpret_cast<const uint32_t*>(list) + (size_t)(k >> 1) * n + i);
}

struct StagePlan {
  int32_t seg_b[kMaxSegs];        // global sorted index of each staged segment
  int32_t seg_len[kMaxSegs];
  int32_t seg_off[kMaxSegs + 1];  // staged offset (prefix of the lengths rounded up to pairs)
  int32_t copied;                 // candidates copied: the sum of the lengths
  int32_t seg_delta[kMaxSegs];    // seg_off - seg_b: a staged candidate sits at its sorted index + delta
  int32_t col0;                   // first column (x*ny + y) of the CTA
  int32_t ncols;                  // 1 .. kMaxCols; 0 = read from global memory
};

// Warp 0 plans the CTA's staging: the columns its particles occupy and, per
// column, the candidate rows over the z cells its particles' windows can
// reach (rz cells beyond the particles' own).
__device__ __forceinline__ void plan_stage(const SceneDev* S, const int32_t* __restrict__ start,
                                           const int32_t* __restrict__ keys, const Tile& tl, StagePlan& sp) {
  const int lane = threadIdx.x & 31;
  const CellCoord a = cell_of_key(S, __ldg(keys + tl.begin));
  const CellCoord b = cell_of_key(S, __ldg(keys + tl.end - 1));
  const int nx = S->dims[0], ny = S->dims[1], nz = S->dims[2];
  const int colA = a.x * ny + a.y, colB = b.x * ny + b.y;
  const int ncols = colB - colA + 1;
  const int R = S->rz;
  int len = 0, gb = 0;
  if (ncols <= kMaxCols && lane < 9 * ncols) {
    const int g = lane / 9, r = lane % 9;
    const int col = colA + g;
    const int cx = (int)(((unsigned long long)(uint32_t)col * S->my) >> S->sy), cy = col - cx * ny;
    const int zlo = g == 0 ? max(a.z - R, 0) : 0;
    const int zhi = (g == ncols - 1) ? min(b.z + R, nz - 1) : nz - 1;
    const int x = cx + r / 3 - 1, y = cy + r % 3 - 1;
    if (x >= 0 && x < nx && y >= 0 && y < ny) {
      const int row = S->coff + (x * ny + y) * nz;
      gb = __ldg(start + row + zlo);
      len = __ldg(start + row + zhi + 1) - gb;
    }
  }
  const int padded = (len + 1) & ~1;
  int incl = padded;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  const int copied = __reduce_add_sync(0xffffffffu, len);
  if (lane < kMaxSegs) {
    sp.seg_b[lane] = gb;
    sp.seg_len[lane] = len;
    sp.seg_off[lane] = incl - padded;
    sp.seg_delta[lane] = incl - padded - gb;
  }
  if (lane == 0) {
    sp.seg_off[kMaxSegs] = total;
    sp.copied = copied;
    sp.col0 = colA;
    sp.ncols = (ncols <= kMaxCols && total <= kStageCap) ? ncols : 0;
  }
}

// Candidate test of one row.  DENSITY: q = max(h^2 - r^2, 0) and the sum of
// q^3.  A hit (q > 0 for the radius hit2) is appended to the lane's code
// list, the particle itself included.  CLAMP: the list pointer is clamped
// at the overflow slot after every candidate; rows that cannot reach it
// (the common case, checked once per row) skip the clamp.
template <bool DENSITY, bool CLAMP, class T, class Load>
__device__ __forceinline__ T scan_row_impl(Load load, int len, uint32_t code0, T px, T py, T pz, T hit2,
                                           uint16_t*& hp, uint16_t* hp_end) {
  T part = (T)0;
#pragma unroll 4
  for (int o = 0; o < len; ++o) {
    const float4 pj = load(o);
    const T dx = px - (T)pj.x, dy = py - (T)pj.y, dz = pz - (T)pj.z;
    T q = fma(-dx, dx, hit2);
    q = fma(-dy, dy, q);
    q = fma(-dz, dz, q);
    if (q > (T)0) {  // a miss would add (+0)^3: the sum is unchanged
      if (DENSITY) part = fma(q * q, q, part);
      *hp = (uint16_t)(code0 + (uint32_t)o);
      hp += kNbThreads;
    }
    if (CLAMP) hp = hp < hp_end ? hp : hp_end;
  }
  return part;
}

template <bool DENSITY, class T, class Load>
__device__ __forceinline__ T scan_row(Load load, int len, uint32_t code0, T px, T py, T pz, T hit2,
                                      uint16_t*& hp, uint16_t* hp_end) {
  if (hp + (size_t)len * kNbThreads <= hp_end)
    return scan_row_impl<DENSITY, false, T>(load, len, code0, px, py, pz, hit2, hp, hp_end);
  return scan_row_impl<DENSITY, true, T>(load, len, code0, px, py, pz, hit2, hp, hp_end);
}

// Candidate test of one row for the density pass: the sum of q^3 over the
// hits and the hits themselves as bits of the row window (bit o = candidate
// o; candidates 64 and up are tested and summed but get no bit).  The tests
// only set register bits, so no lane stores anything per candidate.
template <int U, class T, class Load>
__device__ __forceinline__ T scan_row_bits(Load load, int len, T px, T py, T pz, T hit2, RowMask& bits) {
  T part = (T)0;
  uint32_t lo = 0u, hi = 0u;
  for (int c0 = 0; c0 < len; c0 += 32) {
    const int n = min(len - c0, 32);
    uint32_t m = 0u, bit = 1u;
    // Unrolled by 2: a row holds ~12 candidates at C1 (z cells of h/4), so
    // a deeper unroll spends its time in the remainder loop.  With every CTA
    // on this loop the pass took 168 us unrolled by 4, 154 by 2, 165 by 1, 167
    // by 3 and 192 by 8 at C1; staged rows now go through scan_row_pairs.
#pragma unroll U
    for (int o = 0; o < n; ++o) {
      const float4 pj = load(c0 + o);
      const T dx = px - (T)pj.x, dy = py - (T)pj.y, dz = pz - (T)pj.z;
      T q = fma(-dx, dx, hit2);
      q = fma(-dy, dy, q);
      q = fma(-dz, dz, q);
      if (q > (T)0) {  // a miss would add (+0)^3: the sum is unchanged
        part = fma(q * q, q, part);
        m |= bit;
      }
      bit <<= 1;
    }
    if (c0 == 0)
      lo = m;
    else if (c0 == 32)
      hi = m;
  }
  bits = ((RowMask)hi << 32) | lo;
  return part;
}

// The same row in FP64.  A float test against the margin radius (which no
// hit of the double test fails: the margin is 2^-10, the float distance's
// error 2^-22) picks the candidates, and only those run in double, in order;
// the sum and the bits are those of testing every candidate in double.
// FP64 instructions (2 lanes a clock and SM) bound this pass: ~5 for each of
// ~37 candidates a particle instead of ~12 for each of ~130.  With force's
// conversions and division taken out of its pair loop (widen, diff_as, the
// stored 1/rho: ~26 FP64 instructions a pair instead of ~43), the grid,
// density and force of 68,265 particles went from 432 to 209 us.
template <int U, class Load>
__device__ __forceinline__ double scan_row_fp64(Load load, int len, float4 pi, double hit2, float rad2,
                                                RowMask& bits) {
  double part = 0.0;
  uint32_t lo = 0u, hi = 0u;
  for (int c0 = 0; c0 < len; c0 += 32) {
    const int n = min(len - c0, 32);
    uint32_t near = 0u, m = 0u, bit = 1u;
#pragma unroll U
    for (int o = 0; o < n; ++o) {
      const float4 pj = load(c0 + o);
      const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
      if (dx * dx + dy * dy + dz * dz < rad2) near |= bit;
      bit <<= 1;
    }
    while (near) {
      const int o = __ffs((int)near) - 1;
      near &= near - 1u;
      const float4 pj = load(c0 + o);
      const double dx = diff_as(pi.x, pj.x, 0.0), dy = diff_as(pi.y, pj.y, 0.0), dz = diff_as(pi.z, pj.z, 0.0);
      double q = fma(-dx, dx, hit2);
      q = fma(-dy, dy, q);
      q = fma(-dz, dz, q);
      const int top = __double2hiint(q);  // q > 0, tested on its bits
      if (top >= 0 && (top | __double2loint(q)) != 0 && top < 0x7ff00000) {
        part = fma(q * q, q, part);
        m |= 1u << o;
      }
    }
    if (c0 == 0)
      lo = m;
    else if (c0 == 32)
      hi = m;
  }
  bits = ((RowMask)hi << 32) | lo;
  return part;
}

// ---- staged candidates in pairs ----
// The packed float instructions work on two candidates at once and round each
// like the scalar ones, so the stage is rewritten in place: 24 bytes a pair,
// (x0, x1), (y0, y1), (z0, z1).
typedef unsigned long long F2;
constexpr uint32_t kPairBytes = 24;

// Two pairs a thread and round: a round reads 64 bytes a thread and writes 48,
// all of them where this or an earlier round has read.
__device__ __forceinline__ void pair_stage(float4* cand, int pairs) {
  float2* const out = reinterpret_cast<float2*>(cand);
#pragma unroll 1
  for (int q0 = 0; q0 < pairs; q0 += 2 * blockDim.x) {
    float4 a[2], b[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int q = q0 + k * blockDim.x + threadIdx.x;
      if (q < pairs) a[k] = cand[2 * q], b[k] = cand[2 * q + 1];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int q = q0 + k * blockDim.x + threadIdx.x;
      if (q < pairs) {
        out[3 * q] = make_float2(a[k].x, b[k].x);
        out[3 * q + 1] = make_float2(a[k].y, b[k].y);
        out[3 * q + 2] = make_float2(a[k].z, b[k].z);
      }
    }
  }
  // a later tile's bulk copies write the same words
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ F2 f2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 f2_get(F2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// scan_row_bits over staged candidates [o0, o0 + len) of the stage at `stage`,
// in whole pairs: what the first and the last pair may hold besides (a row's
// candidate outside the window, or the filler) is out of reach.  The distance
// is formed with its sign turned, nq = r^2 - h^2, so that a hit is a set sign
// bit (zeros of an exact cancellation are +0 and the GPU's NaNs have none) and
// goes into the mask with one funnel shift, and min(nq, 0) is what a hit adds
// and nothing for a miss: 17 instructions a pair in place of 26, and the same
// bits.  At 1M particles the pass went from 128M warp instructions and 129 us
// to 109M and 122 (issue still bounds it, at 73%); unrolled by 1 or 4 three
// interleaved sims' steps take 1.5% longer.
__device__ __forceinline__ float scan_row_pairs(uint32_t stage, int o0, int len, float4 p, float h, RowMask& bits) {
  const F2 px = f2(p.x, p.x), py = f2(p.y, p.y), pz = f2(p.z, p.z), minus = f2(-1.0f, -1.0f);
  const float nh = -(h * h);
  const F2 nh2 = f2(nh, nh);
  const int odd = o0 & 1;
  uint32_t a = stage + kPairBytes * (uint32_t)(o0 >> 1);
  int left = (len + odd + 1) >> 1;
  float part = 0.0f;
  uint32_t lo = 0u, hi = 0u, top = 0u;
  for (int c0 = 0; left > 0; c0 += 32, left -= 16) {
    const int n = min(left, 16);
    uint32_t m = 0u;
    const uint32_t end = a + kPairBytes * (uint32_t)n;
#pragma unroll 2
    for (; a < end; a += kPairBytes) {
      F2 xj, yj, zj;
      asm("ld.shared.b64 %0, [%1];" : "=l"(xj) : "r"(a));
      asm("ld.shared.b64 %0, [%1];" : "=l"(yj) : "r"(a + 8u));
      asm("ld.shared.b64 %0, [%1];" : "=l"(zj) : "r"(a + 16u));
      const F2 dx = f2_fma(xj, minus, px), dy = f2_fma(yj, minus, py), dz = f2_fma(zj, minus, pz);
      const float2 nq = f2_get(f2_fma(dz, dz, f2_fma(dy, dy, f2_fma(dx, dx, nh2))));
      m = __funnelshift_l(__float_as_uint(nq.x), m, 1);
      m = __funnelshift_l(__float_as_uint(nq.y), m, 1);
      const float t0 = fminf(nq.x, 0.0f), t1 = fminf(nq.y, 0.0f);
      part = fmaf(t0 * t0, -t0, part);
      part = fmaf(t1 * t1, -t1, part);
    }
    m = __brev(m) >> (32 - 2 * n);
    if (c0 == 0)
      lo = m;
    else if (c0 == 32)
      hi = m;
    else if (c0 == 64)
      top = m;
  }
  bits = ((RowMask)hi << 32) | lo;
  if (odd) bits = (bits >> 1) | ((RowMask)top << 63);
  return part;
}

// One candidate row in the precision P (hit2 = h^2, rad2 >= its float
// rounding with a margin).
template <int P, int U, class Load>
__device__ __forceinline__ Real<P> scan_row_prec(Load load, int len, float4 pi, Real<P> hit2, float rad2,
                                                 RowMask& bits) {
  if constexpr (P == CWA_PREC_FP64)
    return scan_row_fp64<U>(load, len, pi, hit2, rad2, bits);
  else
    return scan_row_bits<U, float>(load, len, pi.x, pi.y, pi.z, hit2, bits);
}

// Candidate scan.  MODE_DENSITY (per-step mode): radius h, density + this
// step's row masks.  MODE_LIST (Verlet mode, only when the rebuild flag is
// up): radius h (1 + skin), the Verlet list and the rebuild positions.
constexpr int MODE_DENSITY = 0;
constexpr int MODE_LIST = 1;

// Shared memory of the candidate scan.
template <int MODE>
struct ScanShared {
  static constexpr bool kCanStage = MODE == MODE_DENSITY;
  __align__(128) float4 cand[kCanStage ? kStageCap : 1];
  // the Verlet list build stages its codes (+ the overflow slot); the
  // density pass keeps its hits in registers
  uint16_t hit[MODE == MODE_LIST ? kMaxVerlet + 1 : 1][kNbThreads];
  StagePlan sp;
  __align__(8) uint64_t bar;
};

// One tile of the candidate scan.  Stages the tile's rows (bulk copies that
// complete phase `parity` of the CTA's barrier) and scans them.  Returns 1
// when the tile was staged (a barrier phase was used), plus 2 when the
// staging wait timed out (then nothing was computed).  Contains CTA-wide
// barriers: every thread of the CTA calls it.
template <int P, int MODE>
__device__ __forceinline__ int scan_tile(
    ScanShared<MODE>& sh, const Tile tl, uint32_t parity, const float4* __restrict__ pos,
    const int32_t* __restrict__ start, const int32_t* __restrict__ keys, const SceneDev* __restrict__ scenes,
    const float* __restrict__ wave, float2* __restrict__ rho_p, uint16_t* __restrict__ list,
    int32_t* __restrict__ list_cnt, RowMask* __restrict__ masks, float4* __restrict__ xref, int32_t n_total,
    int32_t* status, int32_t allow_stage, const float4* __restrict__ vel, PairRec* __restrict__ pairs,
    double* __restrict__ irho) {
  using T = Real<P>;
  constexpr int kCap = kMaxVerlet;  // the Verlet list build's codes per particle
  // The list build (rare: Verlet rebuilds only) reads candidates from global
  // memory, which keeps its static shared memory under 48 KB.
  constexpr bool kCanStage = ScanShared<MODE>::kCanStage;
  constexpr bool kPairs = kCanStage && P != CWA_PREC_FP64;  // the stage is rewritten in pairs (scan_row_pairs)
  float4* const s_cand = sh.cand;
  StagePlan& sp = sh.sp;
  const SceneDev* S = scenes + tl.scene;
  if (threadIdx.x < 32) plan_stage(S, start, keys, tl, sp);
  __syncthreads();
  const bool staged = kCanStage && allow_stage && sp.ncols > 0;
  if (staged && threadIdx.x < 32) {
    // lane s: segment s (at most 27: one warp issues all the copies at once)
    const int s = threadIdx.x, len = s < 9 * sp.ncols ? sp.seg_len[s] : 0;
    // an odd segment's last pair is filled up with a candidate out of reach,
    // before thread 0 arms the barrier: its arrival releases the lanes' stores
    // to the threads that wait on the barrier
    const float far = __int_as_float(0x7f800000);
    if (kPairs && (len & 1)) s_cand[sp.seg_off[s] + len] = make_float4(far, far, far, 0.0f);
    __syncwarp();
    if (s == 0) mbar_expect_tx(&sh.bar, (uint32_t)sp.copied * 16u);
    __syncwarp();
    if (len > 0) bulk_g2s(&s_cand[sp.seg_off[s]], pos + sp.seg_b[s], (uint32_t)len * 16u, &sh.bar);
  }
  bool ready = true;
  if (staged && !mbar_wait_bounded(&sh.bar, parity)) {
    ready = false;
    if (threadIdx.x == 0) atomicOr(status, kStatusTimeout);
    mbar_wait_bounded(&sh.bar, parity);  // let copies in flight land before the CTA moves on
  }
  const int used = (staged ? 1 : 0) | (ready ? 0 : 2);
  if (kPairs && staged) {
    pair_stage(s_cand, sp.seg_off[kMaxSegs] >> 1);
    __syncthreads();
  }
  const int i = tl.begin + threadIdx.x;
  if (i >= tl.end || !ready) return used;

  const float4 pi = __ldg(pos + i);
  const T hh = (T)S->h;
  const T hit2 = MODE == MODE_DENSITY ? hh * hh : (T)S->hl2;
  const T px = pi.x, py = pi.y, pz = pi.z;
  const CellCoord c = cell_of_key(S, __ldg(keys + i));
  int b[9], e[9], base[9];
  row_ranges(S, start, pi, c, S->hl2, b, e);
  row_bases(S, start, c, base);
  const int g = staged ? c.x * S->dims[1] + c.y - sp.col0 : 0;
  uint16_t* const hit_col = &sh.hit[0][threadIdx.x];
  uint16_t* const hp_end = hit_col + kCap * kNbThreads;  // the overflow slot (list build)
  uint16_t* hp = hit_col;
  Sum<P> acc;
  bool overflow = false;
  int hits = 0;  // rows with a nonzero mask (bit r)
  if (MODE == MODE_DENSITY) {
    // In a dense spot the candidates below a window can push it past its
    // row's 64 bits; such a particle's masks count from the windows' own
    // starts (kWindowMasks), which force recomputes.
    int reach = 0;
#pragma unroll
    for (int r = 0; r < 9; ++r) reach = max(reach, e[r] - base[r]);
    if (reach > kMaskBits) {
      hits = kWindowMasks;
#pragma unroll
      for (int r = 0; r < 9; ++r) base[r] = b[r];
    }
  }
  // One row's hits as bits relative to the row's base, and its sum.
  auto row_done = [&](int r, int off0, int len, RowMask bits, T part) {
    overflow |= off0 + len > kMaskBits;
    const RowMask m = off0 < kMaskBits ? bits << off0 : 0u;
    // every row is stored (whole sectors: skipping the zero rows would make
    // each store a partial-sector write that DRAM reads back to merge);
    // force reads only the rows the bitmap names
    masks[(size_t)r * n_total + i] = m;
    if (m != 0u) hits |= 1 << r;
    acc.add(part);
  };
  if (MODE == MODE_DENSITY && staged) {
#pragma unroll
    for (int r = 0; r < 9; ++r) {
      int len = e[r] - b[r];
      const int so = b[r] + sp.seg_delta[g * 9 + r];
      if (CWA_DCHECK_FAILED(len == 0 || (g >= 0 && g < sp.ncols && so >= 0 && so + len <= sp.seg_off[kMaxSegs]),
                            status))
        len = 0;
      RowMask bits = 0u;
      T part = (T)0;
      if (len > 0) {
        if (kPairs) {
          part = scan_row_pairs(smem_u32(s_cand), so, len, pi, S->h, bits);
        } else {
          const uint32_t a0 = smem_u32(s_cand + so);
          part = scan_row_prec<P, 2>([&](int o) { return lds128(a0 + 16u * (uint32_t)o); }, len, pi, hit2, S->hs2,
                                     bits);
        }
      }
      row_done(r, b[r] - base[r], len, bits, part);
    }
  } else if (MODE == MODE_DENSITY) {
    // A CTA that spans too many columns or candidates to stage, rolled up.
    // With both forms in each of the nine unrolled rows the pass took 123 us
    // and not 117 at 1M particles, and ten steps of three interleaved sims
    // 3585 us and not 3010: this way the kernel has 72 registers, and seven
    // CTAs a SM where there were eight leave more of the SM's memory as L1 to
    // the force CTAs of another sim (asking for the shared memory of eight
    // brings 3690 us back).
    const RowWindows w(S, pi, c, S->hl2);
    const int zb = max(c.z - S->rz, 0);
#pragma unroll 1
    for (int r = 0; r < 9; ++r) {
      int rb, re;
      w.range(S, start, c, r, rb, re);
      int len = re - rb;
      if (CWA_DCHECK_FAILED(len == 0 || (rb >= 0 && len > 0 && re <= n_total), status)) len = 0;
      const int rbase = hits & kWindowMasks ? rb : row_valid(S, c, r) ? __ldg(start + row_id(S, c, r) + zb) : 0;
      const float4* cand = pos + rb;
      RowMask bits = 0u;
      T part = (T)0;
      if (len > 0) part = scan_row_prec<P, 2>([&](int o) { return __ldg(cand + o); }, len, pi, hit2, S->hs2, bits);
      row_done(r, rb - rbase, len, bits, part);
    }
  } else {
#pragma unroll
    for (int r = 0; r < 9; ++r) {
      int len = e[r] - b[r];
      if (CWA_DCHECK_FAILED(len == 0 || (b[r] >= 0 && len > 0 && e[r] <= n_total), status)) len = 0;
      const int off0 = b[r] - base[r];
      const float4* cand = pos + b[r];
      overflow |= off0 + len > kRowCodeMax;
      const uint32_t code0 = ((uint32_t)r << kRowCodeBits) + (uint32_t)off0;
      if (len > 0)
        scan_row<false, T>([&](int o) { return __ldg(cand + o); }, len, code0, px, py, pz, hit2, hp, hp_end);
    }
  }
  if (MODE == MODE_LIST) {
    // Coalesced list write: the pair (k, k+1) of every lane is one 128-byte
    // store per warp.  (Row k+1 <= kCap exists: s_hit has the overflow row.)
    const int cnt = (int)(hp - hit_col) / kNbThreads;
    overflow |= cnt >= kCap;
    uint32_t* const list32 = reinterpret_cast<uint32_t*>(list);
    for (int k = 0; k < cnt; k += 2)
      list32[(size_t)(k >> 1) * n_total + i] =
          (uint32_t)hit_col[k * kNbThreads] | ((uint32_t)hit_col[(k + 1) * kNbThreads] << 16);
    list_cnt[i] = overflow ? kCap + 1 : cnt;
    xref[i] = pi;
  } else {
    list_cnt[i] = overflow ? -1 : hits;
    const T rho_t = (P == CWA_PREC_FP64 ? (T)S->c_poly6_d : (T)S->c_poly6) * acc.get();
    const float2 rp = eos(S, (float)rho_t, pi, wave);
    rho_p[i] = rp;
    write_pair_rec<P>(pairs, irho, vel, i, pi, rp);
  }
  return used;
}

// The candidate scan over the tile list, one CTA a tile; or (queue set,
// density mode only) as the work-queue form: resident CTAs take tile
// numbers from the counter *queue and scan tiles[order[t]] until the
// n_tiles of the launch are taken.
template <int P, int MODE, int MINB, bool WQ>
__global__ void __launch_bounds__(kNbThreads, MINB)
    k_scan_cands(const float4* __restrict__ pos, const int32_t* __restrict__ start,
                 const int32_t* __restrict__ keys, const Tile* __restrict__ tiles,
                 const SceneDev* __restrict__ scenes, const float* __restrict__ wave,
                 float2* __restrict__ rho_p, uint16_t* __restrict__ list, int32_t* __restrict__ list_cnt,
                 RowMask* __restrict__ masks, float4* __restrict__ xref, int32_t n_total, int32_t* status,
                 const int32_t* __restrict__ flag, int32_t allow_stage, const float4* __restrict__ vel,
                 PairRec* __restrict__ pairs, double* __restrict__ irho, const int32_t* __restrict__ order,
                 int32_t* queue, int32_t n_tiles) {
  __shared__ ScanShared<MODE> sh;
  __shared__ int32_t s_next;
  if (MODE == MODE_LIST && flag && __ldg(flag) == 0) return;  // no rebuild this step
  if (threadIdx.x == 0) mbar_init(&sh.bar, 1);
  if constexpr (!WQ || MODE != MODE_DENSITY) {
    scan_tile<P, MODE>(sh, tiles[blockIdx.x], 0u, pos, start, keys, scenes, wave, rho_p, list, list_cnt, masks,
                       xref, n_total, status, allow_stage, vel, pairs, irho);
    return;
  }
  uint32_t parity = 0u;
  for (;;) {
    if (threadIdx.x == 0) s_next = atomicAdd(queue, 1);
    __syncthreads();  // also: every thread is done with the previous tile's stage and plan
    const int t = s_next;
    __syncthreads();  // s_next read by all before thread 0 may take the next number
    if (t >= n_tiles) break;
    const int used = scan_tile<P, MODE>(sh, tiles[__ldg(order + t)], parity, pos, start, keys, scenes, wave, rho_p,
                                        list, list_cnt, masks, xref, n_total, status, allow_stage, vel, pairs, irho);
    if (__syncthreads_or(used & 2)) break;  // a staging wait timed out (status set): stop taking tiles
    if (used & 1) parity ^= 1u;
  }
}

// Verlet density: walks the particle's list (pairs within h (1 + skin) at
// the last rebuild), accumulates the poly6 sum over r < h in groups of 8
// (partials folded into the precision mode's accumulator), and writes this
// step's row masks for force.  A particle whose Verlet list overflowed
// rescans the rows of its rebuild cell.
template <int P>
__global__ void __launch_bounds__(kNbThreads, 8)
    k_rho_list(const float4* __restrict__ pos, const int32_t* __restrict__ start,
               const int32_t* __restrict__ keys, const Tile* __restrict__ tiles,
               const SceneDev* __restrict__ scenes, const float* __restrict__ wave,
               float2* __restrict__ rho_p, const uint16_t* __restrict__ vlist,
               const int32_t* __restrict__ vcnt, RowMask* __restrict__ nbm, int32_t* __restrict__ nbr_cnt,
               int32_t n_total, const float4* __restrict__ vel, PairRec* __restrict__ pairs,
               double* __restrict__ irho) {
  using T = Real<P>;
  __shared__ int32_t s_rb[9][kNbThreads];
  __shared__ RowMask s_m[kNbRows][kNbThreads];  // this step's row masks
  const Tile tl = tiles[blockIdx.x];
  const int i = tl.begin + threadIdx.x;
  if (i >= tl.end) return;
  const SceneDev* S = scenes + tl.scene;
  const float4 pi = __ldg(pos + i);
  const T hh = (T)S->h;
  const T h2 = hh * hh;
  const T px = pi.x, py = pi.y, pz = pi.z;
  const CellCoord c = cell_of_key(S, __ldg(keys + i));
  int base[9];
  row_bases(S, start, c, base);
  Sum<P> acc;
  bool overflow = false;
  const int vn = __ldg(vcnt + i);
#pragma unroll
  for (int r = 0; r < kNbRows; ++r) s_m[r][threadIdx.x] = 0u;
  // candidate j at offset off of row r (r < 9): a hit sets its row-mask
  // bit, or marks the particle overflowed when off is past the mask's last bit
  auto test = [&](int j, int r, uint32_t off) {
    const float4 pj = __ldg(pos + j);
    const T dx = px - (T)pj.x, dy = py - (T)pj.y, dz = pz - (T)pj.z;
    T q = fma(-dx, dx, h2);
    q = fma(-dy, dy, q);
    q = fma(-dz, dz, q);
    const T qp = q > (T)0 ? q : (T)0;
    if (q > (T)0) {
      if (off < (uint32_t)kMaskBits)
        s_m[r][threadIdx.x] |= (RowMask)1u << off;
      else
        overflow = true;
    }
    return qp * qp * qp;
  };
  if (vn <= kMaxVerlet) {
#pragma unroll
    for (int r = 0; r < 9; ++r) s_rb[r][threadIdx.x] = base[r];
    for (int k0 = 0; k0 < vn; k0 += 8) {
      uint32_t code[8];
#pragma unroll
      for (int u = 0; u < 8; u += 2) {
        const uint32_t w = k0 + u < vn ? code_pair(vlist, k0 + u, i, n_total) : 0u;
        code[u] = w & 0xFFFFu;
        code[u + 1] = k0 + u + 1 < vn ? w >> 16 : 0u;
      }
      T part = (T)0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int rr = (int)(code[u] >> kRowCodeBits);
        const uint32_t off = code[u] & (kRowCodeMax - 1);
        const int j = s_rb[rr][threadIdx.x] + (int)off;
        if (k0 + u < vn) part += test(j, rr, off);
      }
      acc.add(part);
    }
  } else {
    // the rows of the rebuild cell over every z cell a pair within
    // h (1 + skin) could occupy; hits take bits against the same bases
    const int z1 = min(c.z + S->rz, S->dims[2] - 1);
#pragma unroll
    for (int r = 0; r < 9; ++r) {
      if (!row_valid(S, c, r)) continue;
      const int e = __ldg(start + row_id(S, c, r) + z1 + 1);
      T part = (T)0;
      for (int j = base[r]; j < e; ++j) part += test(j, r, (uint32_t)(j - base[r]));
      acc.add(part);
    }
  }
  int rows = 0;  // rows with a nonzero mask (bit r)
#pragma unroll
  for (int r = 0; r < kNbRows; ++r) {
    const RowMask m = s_m[r][threadIdx.x];
    nbm[(size_t)r * n_total + i] = m;
    if (m != 0u) rows |= 1 << r;
  }
  nbr_cnt[i] = overflow ? -1 : rows;
  const T rho_t = (P == CWA_PREC_FP64 ? (T)S->c_poly6_d : (T)S->c_poly6) * acc.get();
  const float2 rp = eos(S, (float)rho_t, pi, wave);
  rho_p[i] = rp;
  write_pair_rec<P>(pairs, irho, vel, i, pi, rp);
}

// The force a particle stores: pressure + viscosity sums (already scaled,
// fpr / fvr) plus gravity, and for REFERENCE_3D the shader's crest, torque,
// drag and wave-normal terms (force_comp.glsl:90-114).
__device__ __forceinline__ float4 force_out(const SceneDev* S, int i, float4 pi, float4 vi, float rho,
                                            const float fpr[3], const float fvr[3], const float4* force,
                                            const float* __restrict__ wave) {
  float4 out;
  if (S->preset == CWA_PRESET_REFERENCE_3D) {
    float4 fprev = force[i];
    float vs = S->visc;
    if (pi.y > S->crest) {
      fprev.x /= 0.25f;
      fprev.y /= 0.25f;
      fprev.z /= 0.25f;
      fprev.w /= 0.25f;
      vs *= 0.5f;
    }
    const float* u = wave + S->woff;
    const int W = S->nx, Hn = S->nz;
    const float s = uv_s(S, pi.x), t = uv_t(S, pi.z);
    const float H = sample_height(u, W, Hn, s, t);
    const float tq[3] = {0.25f * (pi.y * fprev.z - pi.z * fprev.y), 0.25f * (pi.z * fprev.x - pi.x * fprev.z),
                         0.25f * (pi.x * fprev.y - pi.y * fprev.x)};
    // WaveVelocity (:117-128) and WaveNormal (:130-139)
    const float hx = sample_height(u, W, Hn, s + 0.01f, t);
    const float hy = sample_height(u, W, Hn, s, t + 0.01f);
    const float wv[3] = {(hx - H) / S->dt, (hy - H) / S->dt, (hx - hy) / 0.01f};
    const float hR = sample_height(u, W, Hn, s + 1.0f, t) - H;
    const float hT = sample_height(u, W, Hn, s, t + 1.0f) - H;
    const float nrm[3] = {hR, hT, -1.0f};
    const float vv[3] = {vi.x, vi.y, vi.z};
    float f[3];
#pragma unroll
    for (int c2 = 0; c2 < 3; ++c2) {
      const float drag = -0.25f * (vv[c2] - wv[c2]);
      const float wf = -H * nrm[c2] * 0.5f;
      f[c2] = fpr[c2] + fvr[c2] * vs + rho * S->g[c2] + tq[c2] + drag + wf;
    }
    out = make_float4(f[0], f[1], f[2], fprev.w);
  } else {
    out = make_float4(fpr[0] + fvr[0] * S->visc + rho * S->g[0], fpr[1] + fvr[1] * S->visc + rho * S->g[1],
                      fpr[2] + fvr[2] * S->visc + rho * S->g[2], 0.0f);
  }
  return out;
}

// Three-component sum in the precision mode: COMPENSATED adds pair terms
// in float into a partial that the caller folds into a two-sum accumulator
// after every group of 8 pairs (cascaded summation); FP32 is plain; FP64 is
// double.
template <int P>
struct Acc3 {
  Sum<P> x, y, z;
  Real<P> px = 0, py = 0, pz = 0;
  __device__ __forceinline__ void add(Real<P> a, Real<P> b, Real<P> c) {
    if (P == CWA_PREC_COMPENSATED) {
      px += a;
      py += b;
      pz += c;
    } else {
      x.add(a);
      y.add(b);
      z.add(c);
    }
  }
  __device__ __forceinline__ void flush() {
    if (P == CWA_PREC_COMPENSATED) {
      x.add(px);
      y.add(py);
      z.add(pz);
      px = py = pz = 0;
    }
  }
};

// One particle's pair sums of the force pass: spiky pressure gradient and
// viscosity Laplacian over neighbours j.
template <int P>
struct PairSums {
  using T = Real<P>;
  float px, py, pz;
  T vx, vy, vz, pres, h;
  Acc3<P> fp, fv;
  __device__ __forceinline__ void init(const SceneDev* S, float4 pi, float4 vi, float p) {
    px = pi.x;
    py = pi.y;
    pz = pi.z;
    vx = vi.x;
    vy = vi.y;
    vz = vi.z;
    pres = p;
    h = (T)S->h;
  }
  // xj, vj: the neighbour's gather records
  __device__ __forceinline__ void pair(float4 xj, float4 vj, T irho) {
    const T z = (T)0;
    const T dx = diff_as(px, xj.x, z), dy = diff_as(py, xj.y, z), dz = diff_as(pz, xj.z, z);
    const T r2 = dx * dx + dy * dy + dz * dz;
    const T inv_r = r2 > (T)0 ? inv_sqrt(r2) : (T)0;  // normalize(0) := 0
    const T r = r2 * inv_r;
    const T hr = h - r;
    const T sp = (pres + widen_as(xj.w, z)) * irho * hr * hr * inv_r;
    fp.add(sp * dx, sp * dy, sp * dz);
    const T sv = irho * hr;
    fv.add(sv * (widen_as(vj.x, z) - vx), sv * (widen_as(vj.y, z) - vy), sv * (widen_as(vj.z, z) - vz));
  }
  __device__ __forceinline__ void flush() {
    fp.flush();
    fv.flush();
  }
};

// The arrays a pair's neighbour data comes from (the density pass's records)
// and the positions.
struct PairArrays {
  const float4* __restrict__ pos;
  const PairRec* __restrict__ pairs;
  const double* __restrict__ irho;
};

// 1/rho of neighbour j in the precision P.
template <int P>
__device__ __forceinline__ Real<P> inv_rho(const PairArrays& a, float4 vj, int j) {
  if constexpr (P == CWA_PREC_FP64)
    return __ldg(a.irho + j);
  else
    return vj.w;
}

// Adds the pairs of the hits in m (bit b = candidate j0 + b), lowest bit
// first; U hits' gathers are in flight at a time.
template <int P, int U, class M>
__device__ __forceinline__ void add_hits(PairSums<P>& s, const PairArrays& a, int j0, M m) {
#pragma unroll 1
  while (m) {
    int js[U];
    int k = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      js[u] = j0 + (m ? __ffsll((long long)m) - 1 : 0);
      k += m != 0;
      m &= m - 1;
    }
    float4 xj[U], vj[U];
    Real<P> ir[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      load_pair(a.pairs + js[u], xj[u], vj[u]);
      ir[u] = inv_rho<P>(a, vj[u], js[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < k) s.pair(xj[u], vj[u], ir[u]);
  }
}

// Candidate row r of a particle in a dense spot (kWindowMasks, or -1: a row
// window of more than 64 candidates).  With masks, their bits count from the
// row window's start; without, the window is tested again, 32 candidates at a
// time with U loads in flight.  The caller folds the sums once a row.
// Such particles are few but sit on the pass's critical path: testing each
// candidate and gathering its hit at once, over every z cell a neighbour
// could occupy, cost one dependent round trip a candidate and kept single
// warps running 40 us past the others (force 160 -> 127 us in the 1M-particle
// run while the sheet of surface particles is dense).
template <int P, int U>
__device__ __forceinline__ void dense_row(PairSums<P>& s, const PairArrays& a, const SceneDev* S,
                                          const int32_t* __restrict__ start, const RowWindows& w, CellCoord c, int i,
                                          int r, int cnt, const RowMask* __restrict__ nbm, int32_t n_total) {
  using T = Real<P>;
  int b, e;
  w.range(S, start, c, r, b, e);
  if (cnt >= 0) {
    RowMask m = (cnt >> r) & 1 ? __ldg(nbm + (size_t)r * n_total + i) : (RowMask)0u;
    if (r == 4) m &= ~((RowMask)1u << (i - b));  // the particle itself
    add_hits<P, U>(s, a, b, m);
    return;
  }
  const T h2 = s.h * s.h;
#pragma unroll 1
  for (; b < e; b += 32) {
    const int n = min(e - b, 32);
    uint32_t m = 0u;
#pragma unroll 1
    for (int o = 0; o < n; o += U) {
      float4 pj[U];
#pragma unroll
      for (int u = 0; u < U; ++u) pj[u] = __ldg(a.pos + b + min(o + u, n - 1));
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const T dx = diff_as(s.px, pj[u].x, h2), dy = diff_as(s.py, pj[u].y, h2), dz = diff_as(s.pz, pj[u].z, h2);
        T q = fma(-dx, dx, h2);
        q = fma(-dy, dy, q);
        q = fma(-dz, dz, q);
        if (q > (T)0 && o + u < n && b + o + u != i) m |= 1u << (o + u);
      }
    }
    add_hits<P, U>(s, a, b, m);
  }
}

// force: spiky pressure gradient + viscosity Laplacian over the step's hits
// (the row masks), then the preset's extra terms.  Neighbour data comes from
// global memory (L1-resident for the most part: a CTA's particles share their
// candidate rows).  Staging the rows' records in shared memory, as the
// candidate scan does, measured slower here: 48 KB of stage per CTA halves
// the resident warps this latency-bound loop needs.
template <int P>
__device__ __forceinline__ void force_tile(
    RowMask (&s_w)[kNbRows][kNbThreads], int32_t (&s_jb)[kNbRows][kNbThreads], const Tile tl,
    const float4* __restrict__ pos, const float2* __restrict__ rho_p,
    const int32_t* __restrict__ start, const int32_t* __restrict__ keys, const SceneDev* __restrict__ scenes,
    const float* __restrict__ wave, float4* __restrict__ force, const RowMask* __restrict__ nbm,
    const int32_t* __restrict__ nbr_cnt, int32_t n_total, const PairRec* __restrict__ pairs,
    const double* __restrict__ irho, int32_t* status) {
  using T = Real<P>;
  const SceneDev* S = scenes + tl.scene;
  const int i = tl.begin + threadIdx.x;
  if (i >= tl.end) return;
  // the particle's own position and velocity come from its gather records
  // (the same floats, and lines its neighbours' gathers share)
  float4 pi, vi;
  load_pair(pairs + i, pi, vi);
  const float2 rpi = __ldg(rho_p + i);
  const PairArrays arrays{pos, pairs, irho};
  PairSums<P> s;
  s.init(S, pi, vi, rpi.y);
  const int cnt = __ldg(nbr_cnt + i);
  const CellCoord c = cell_of_key(S, __ldg(keys + i));
  if (cnt >= 0 && !(cnt & kWindowMasks)) {
    int base[9];
    row_bases(S, start, c, base);
    // The row masks hold the particle itself: row 4 (its own column) at bit
    // i - base[4], cleared here.  Only the nonzero masks are loaded, back to
    // back, and compacted in row order, and
    // hits are then popped in row then bit order, in groups of 8 whose
    // neighbour indexes are found first so the gathers overlap.
    int nw = 0, left = 0;
#pragma unroll
    for (int r = 0; r < kNbRows; ++r) {
      // cnt: the rows with hits, as bits; the zero rows are not read
      RowMask m = (cnt >> r) & 1 ? __ldg(nbm + (size_t)r * n_total + i) : (RowMask)0u;
      if (r == 4) m &= ~((RowMask)1u << (i - base[4]));
      if (m) {
        s_w[nw][threadIdx.x] = m;
        s_jb[nw][threadIdx.x] = base[r];
        ++nw;
      }
      left += __popcll(m);
    }
    int wi = 0;
    RowMask cw = nw > 0 ? s_w[0][threadIdx.x] : 0u;
    int jb = nw > 0 ? s_jb[0][threadIdx.x] : 0;
    for (int k0 = 0; k0 < left; k0 += 8) {
      int js[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        js[u] = -1;
        if (k0 + u < left) {
          if (cw == 0u) {  // the next mask (every compacted mask holds a hit)
            ++wi;
            cw = s_w[wi][threadIdx.x];
            jb = s_jb[wi][threadIdx.x];
          }
          js[u] = jb + __ffsll((long long)cw) - 1;
          cw &= cw - 1u;
        }
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (js[u] >= 0 && !CWA_DCHECK_FAILED(js[u] < n_total, status)) {
          float4 xj, vj;
          load_pair(pairs + js[u], xj, vj);
          s.pair(xj, vj, inv_rho<P>(arrays, vj, js[u]));
        }
      s.flush();
    }
  } else {
    const RowWindows w(S, pi, c, S->hl2);
#pragma unroll 1
    for (int r = 0; r < kNbRows; ++r) {
      dense_row<P, 2>(s, arrays, S, start, w, c, i, r, cnt, nbm, n_total);
      s.flush();
    }
  }
  s.flush();
  const T cg = P == CWA_PREC_FP64 ? (T)S->k_grad_d * (T)S->mass : (T)(S->k_grad * S->mass);
  const T cp = (T)0.5 * cg;
  float fpr[3] = {(float)(cp * s.fp.x.get()), (float)(cp * s.fp.y.get()), (float)(cp * s.fp.z.get())};
  float fvr[3] = {(float)(cg * s.fv.x.get()), (float)(cg * s.fv.y.get()), (float)(cg * s.fv.z.get())};
  force[i] = force_out(S, i, pi, vi, rpi.x, fpr, fvr, force, wave);
}

// The force pass over the tile list, one CTA a tile, or (queue set) in the
// work-queue form.
template <int P, int MINB, bool WQ>
__global__ void __launch_bounds__(kNbThreads, MINB)
    k_force(const float4* __restrict__ pos, const float2* __restrict__ rho_p, const int32_t* __restrict__ start,
            const int32_t* __restrict__ keys, const Tile* __restrict__ tiles,
            const SceneDev* __restrict__ scenes, const float* __restrict__ wave, float4* __restrict__ force,
            const RowMask* __restrict__ nbm, const int32_t* __restrict__ nbr_cnt, int32_t n_total,
            const PairRec* __restrict__ pairs, const double* __restrict__ irho,
            int32_t* status, const int32_t* __restrict__ order, int32_t* queue, int32_t n_tiles) {
  // the particle's nonzero row masks and the index of each mask's bit 0
  // (13.8 KB a CTA; 32-bit masks, 9.2 KB a CTA, measured slower: 209 against
  // 143 us over the C1 run).  The default variant runs nine CTAs a SM at 56
  // registers: 135.9 against 139.2 us at eight (64 registers), though nine
  // CTAs' arrays leave the L1 a smaller share of the SM's 256 KB.
  __shared__ RowMask s_w[kNbRows][kNbThreads];
  __shared__ int32_t s_jb[kNbRows][kNbThreads];
  if constexpr (!WQ) {
    force_tile<P>(s_w, s_jb, tiles[blockIdx.x], pos, rho_p, start, keys, scenes, wave, force, nbm, nbr_cnt,
                  n_total, pairs, irho, status);
  } else {
    // work-queue form: resident CTAs take tile numbers from *queue
    __shared__ int32_t s_next[2];
    for (int it = 0;; ++it) {
      if (threadIdx.x == 0) s_next[it & 1] = atomicAdd(queue, 1);
      __syncthreads();  // (two slots: thread 0 refills one while the other is still being read)
      const int t = s_next[it & 1];
      if (t >= n_tiles) break;
      force_tile<P>(s_w, s_jb, tiles[__ldg(order + t)], pos, rho_p, start, keys, scenes, wave, force, nbm,
                    nbr_cnt, n_total, pairs, irho, status);
    }
  }
}

// ---- team forms: several lanes a particle --------------------------------
// A scene of a few tens of thousands of particles leaves most of the GPU
// idle with one thread a particle: every pass lasts as long as its longest
// thread.  Here T neighbouring lanes share a particle.  The candidate rows
// are dealt to the lanes (row r to lane r mod T), and so are force's groups of
// 8 hits; every row's and every group's partial sum is formed by one lane in
// the order of the one-thread forms, and the partials are folded into the
// accumulator in the same order on every lane, so the results are the same
// bits.  No staging: the lanes read candidates through L1, with several loads
// in flight.  What bounds them is still latency; they trade total issue for a
// third of the longest thread's chain: the reference scene's step (20,480
// particles, walls with ~100 particles a cell) went from 88 to 51 us alone
// and from 34 to 21 us with three sims interleaved, at four lanes.  Launching
// them as programmatic dependents measured slower (22 against 18.8 us a step
// at 18,816 particles with three sims interleaved).
constexpr int kTeamLanes = 4;

template <int T>
struct Team {
  static constexpr int kRounds = (kNbRows + T - 1) / T;
  int lane;        // this thread's place in its team
  unsigned mask;   // the team's lanes of the warp
  __device__ __forceinline__ Team() {
    const int l = threadIdx.x & 31;
    lane = l & (T - 1);
    mask = (T == 32 ? 0xffffffffu : ((1u << T) - 1u)) << (l - lane);
  }
  template <class V>
  __device__ __forceinline__ V from(V v, int k) const {
    return __shfl_sync(mask, v, k, T);
  }
  __device__ __forceinline__ int max_all(int v) const {
#pragma unroll
    for (int o = 1; o < T; o <<= 1) v = max(v, __shfl_xor_sync(mask, v, o, T));
    return v;
  }
  __device__ __forceinline__ int or_all(int v) const {
#pragma unroll
    for (int o = 1; o < T; o <<= 1) v |= __shfl_xor_sync(mask, v, o, T);
    return v;
  }
  __device__ __forceinline__ int sum_all(int v) const {
#pragma unroll
    for (int o = 1; o < T; o <<= 1) v += __shfl_xor_sync(mask, v, o, T);
    return v;
  }
};

// The particle of this thread's team, or -1 past the tile's end.  Each tile
// of blockDim.x particles is shared by T consecutive CTAs.
template <int T>
__device__ __forceinline__ int team_particle(const Tile& tl) {
  const int per = blockDim.x / T;
  const int i = tl.begin + (blockIdx.x % T) * per + threadIdx.x / T;
  return i < tl.end ? i : -1;
}

template <int P, int T>
__global__ void __launch_bounds__(kNbThreads)
    k_rho_team(const float4* __restrict__ pos, const int32_t* __restrict__ start, const int32_t* __restrict__ keys,
               const Tile* __restrict__ tiles, const SceneDev* __restrict__ scenes, const float* __restrict__ wave,
               float2* __restrict__ rho_p, int32_t* __restrict__ list_cnt, RowMask* __restrict__ masks,
               int32_t n_total, const float4* __restrict__ vel, PairRec* __restrict__ pairs,
               double* __restrict__ irho, int32_t* status) {
  using R = Real<P>;
  const Tile tl = tiles[blockIdx.x / T];
  const int i = team_particle<T>(tl);
  if (i < 0) return;  // whole teams leave together
  const Team<T> team;
  const SceneDev* S = scenes + tl.scene;
  const float4 pi = __ldg(pos + i);
  const CellCoord c = cell_of_key(S, __ldg(keys + i));
  const R hh = (R)S->h;
  const R h2 = hh * hh;
  const RowWindows w(S, pi, c, S->hl2);
  const int zb = max(c.z - S->rz, 0);
  int b[Team<T>::kRounds], e[Team<T>::kRounds], base[Team<T>::kRounds];
  int reach = 0;
#pragma unroll
  for (int q = 0; q < Team<T>::kRounds; ++q) {
    const int r = q * T + team.lane;
    b[q] = e[q] = base[q] = 0;
    if (r < kNbRows) {
      w.range(S, start, c, r, b[q], e[q]);
      base[q] = row_valid(S, c, r) ? __ldg(start + row_id(S, c, r) + zb) : 0;
      reach = max(reach, e[q] - base[q]);
    }
  }
  int hits = team.max_all(reach) > kMaskBits ? kWindowMasks : 0;
  int overflow = 0;
  R part[Team<T>::kRounds];
#pragma unroll
  for (int q = 0; q < Team<T>::kRounds; ++q) {
    const int r = q * T + team.lane;
    part[q] = (R)0;
    if (r < kNbRows) {
      const int len = e[q] - b[q];
      const int off0 = hits & kWindowMasks ? 0 : b[q] - base[q];
      RowMask bits = 0u;
      if (len > 0 && !CWA_DCHECK_FAILED(b[q] >= 0 && e[q] <= n_total, status)) {
        const float4* cand = pos + b[q];
        part[q] = scan_row_prec<P, 4>([&](int o) { return __ldg(cand + o); }, len, pi, h2, S->hs2, bits);
      }
      overflow |= off0 + len > kMaskBits;
      const RowMask m = off0 < kMaskBits ? bits << off0 : 0u;
      masks[(size_t)r * n_total + i] = m;
      if (m != 0u) hits |= 1 << r;
    }
  }
  hits = team.or_all(hits);
  overflow = team.or_all(overflow);
  Sum<P> acc;
#pragma unroll
  for (int r = 0; r < kNbRows; ++r) acc.add(team.from(part[r / T], r % T));
  if (team.lane != 0) return;
  list_cnt[i] = overflow ? -1 : hits;
  const R rho_t = (P == CWA_PREC_FP64 ? (R)S->c_poly6_d : (R)S->c_poly6) * acc.get();
  const float2 rp = eos(S, (float)rho_t, pi, wave);
  rho_p[i] = rp;
  write_pair_rec<P>(pairs, irho, vel, i, pi, rp);
}

// Force in the team form, for the cascaded sums only: their partials (8 hits,
// or a row in a dense spot) split across lanes without changing a rounding;
// the plain and FP64 sums are one chain over all hits.
template <int T>
__global__ void __launch_bounds__(kNbThreads, 6)
    k_force_team(const float4* __restrict__ pos, const float2* __restrict__ rho_p, const int32_t* __restrict__ start,
                 const int32_t* __restrict__ keys, const Tile* __restrict__ tiles,
                 const SceneDev* __restrict__ scenes, const float* __restrict__ wave, float4* __restrict__ force,
                 const RowMask* __restrict__ nbm, const int32_t* __restrict__ nbr_cnt, int32_t n_total,
                 const PairRec* __restrict__ pairs, int32_t* status) {
  constexpr int P = CWA_PREC_COMPENSATED;
  __shared__ RowMask s_w[kNbRows][kNbThreads / T];
  __shared__ int32_t s_jb[kNbRows][kNbThreads / T];
  __shared__ float s_part[kNbThreads][7];  // 7: odd stride, no bank conflicts
  const Tile tl = tiles[blockIdx.x / T];
  const int i = team_particle<T>(tl);
  if (i < 0) return;
  const Team<T> team;
  const int tm = threadIdx.x / T;  // the team's column of the shared arrays
  const SceneDev* S = scenes + tl.scene;
  float4 pi, vi;
  load_pair(pairs + i, pi, vi);
  const float2 rpi = __ldg(rho_p + i);
  const int cnt = __ldg(nbr_cnt + i);
  const CellCoord c = cell_of_key(S, __ldg(keys + i));
  const PairArrays arrays{pos, pairs, nullptr};
  PairSums<P> s;
  s.init(S, pi, vi, rpi.y);
  // Folds the lanes' partials in lane order: lane c keeps the sums of
  // components c, c + T, ... of (pressure xyz, viscosity xyz).
  constexpr int kOwn = (6 + T - 1) / T;
  Sum<P> own[kOwn];
  auto fold = [&]() {
    float* mine = s_part[threadIdx.x];
    mine[0] = s.fp.px;
    mine[1] = s.fp.py;
    mine[2] = s.fp.pz;
    mine[3] = s.fv.px;
    mine[4] = s.fv.py;
    mine[5] = s.fv.pz;
    s.fp.px = s.fp.py = s.fp.pz = s.fv.px = s.fv.py = s.fv.pz = 0.0f;
    __syncwarp(team.mask);
#pragma unroll
    for (int q = 0; q < kOwn; ++q) {
      const int comp = min(q * T + team.lane, 5);
#pragma unroll
      for (int k = 0; k < T; ++k) own[q].add(s_part[tm * T + k][comp]);
    }
    __syncwarp(team.mask);
  };
  if (cnt >= 0 && !(cnt & kWindowMasks)) {
    const int zb = max(c.z - S->rz, 0);
    int left = 0;
#pragma unroll
    for (int q = 0; q < Team<T>::kRounds; ++q) {
      const int r = q * T + team.lane;
      if (r < kNbRows) {
        RowMask m = (cnt >> r) & 1 ? __ldg(nbm + (size_t)r * n_total + i) : (RowMask)0u;
        const int base = row_valid(S, c, r) ? __ldg(start + row_id(S, c, r) + zb) : 0;
        if (r == 4) m &= ~((RowMask)1u << (i - base));  // the particle itself
        s_w[r][tm] = m;
        s_jb[r][tm] = base;
        left += __popcll(m);
      }
    }
    left = team.sum_all(left);
    __syncwarp(team.mask);
    // lane k sums hits 8k .. 8k + 7 of every 8 T, in order
    int wi = -1, skip = 8 * team.lane, jb = 0;
    RowMask cw = 0u;
    for (int g0 = 0; g0 < left; g0 += 8 * T) {
      const int n = min(left - g0 - 8 * team.lane, 8);
      if (n > 0) {
        // walk to this lane's first hit of the round: whole masks, then bits
        for (;;) {
          const int have = __popcll(cw);
          if (skip < have) break;
          skip -= have;
          ++wi;
          cw = s_w[wi][tm];
          jb = s_jb[wi][tm];
        }
        for (; skip > 0; --skip) cw &= cw - 1u;
        int js[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          js[u] = i;
          if (u < n) {
            while (cw == 0u) {
              ++wi;
              cw = s_w[wi][tm];
              jb = s_jb[wi][tm];
            }
            const int j = jb + __ffsll((long long)cw) - 1;
            cw &= cw - 1u;
            if (!CWA_DCHECK_FAILED(j >= 0 && j < n_total, status)) js[u] = j;
          }
        }
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
          float4 xj[4], vj[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            load_pair(pairs + js[h + u], xj[u], vj[u]);
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (h + u < n) s.pair(xj[u], vj[u], vj[u].w);
        }
        skip = 8 * (T - 1);
      }
      fold();
    }
  } else {
    const RowWindows w(S, pi, c, S->hl2);
#pragma unroll 1
    for (int q = 0; q < Team<T>::kRounds; ++q) {
      const int r = q * T + team.lane;
      if (r < kNbRows) dense_row<P, 4>(s, arrays, S, start, w, c, i, r, cnt, nbm, n_total);
      fold();
    }
  }
  float sum[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) sum[k] = team.from(own[k / T].get(), k % T);
  if (team.lane != 0) return;
  const float cg = S->k_grad * S->mass;
  const float cp = 0.5f * cg;
  float fpr[3] = {cp * sum[0], cp * sum[1], cp * sum[2]};
  float fvr[3] = {cg * sum[3], cg * sum[4], cg * sum[5]};
  force[i] = force_out(S, i, pi, vi, rpi.x, fpr, fvr, force, wave);
}

// Grid of a work-queue launch: the CTAs of `kernel` that fit the device at
// once (occupancy x SMs), at most n_tiles.
template <typename K>
int queue_grid(K kernel, int block, int n_tiles) {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0) != cudaSuccess || per_sm < 1)
    return n_tiles;
  return std::min(n_tiles, per_sm * sms);
}

// Launch-bound variants (min CTAs per SM): the register budget trades
// occupancy against loads in flight per warp; the autotuner picks one.
// queue (density mode): the work-queue form, its counter zeroed first.
template <int P, int MODE, int MB>
void scan_launch_one(const NbArgs& a, uint16_t* list, int32_t* cnt, RowMask* masks, float4* xref,
                     const int32_t* flag, int32_t* queue, cudaStream_t st) {
  auto kern = queue ? k_scan_cands<P, MODE, MB, true> : k_scan_cands<P, MODE, MB, false>;
  int grid = a.n_tiles;
  if (queue) {
    cudaMemsetAsync(queue, 0, sizeof(int32_t), st);
    grid = queue_grid(kern, a.tile_size, a.n_tiles);
  }
  kern<<<grid, a.tile_size, 0, st>>>(a.pos, a.start, a.keys, a.tiles, a.scenes, a.wave, a.rho_p, list, cnt, masks,
                                     xref, a.n_total, a.status, flag, a.stage, a.vel, a.pairs, a.irho, a.order,
                                     queue, a.n_tiles);
}

template <int P, int MODE>
void scan_variant(int minb, const NbArgs& a, uint16_t* list, int32_t* cnt, RowMask* masks, float4* xref,
                  const int32_t* flag, int32_t* queue, cudaStream_t st) {
  if (minb >= 8)
    scan_launch_one<P, MODE, 8>(a, list, cnt, masks, xref, flag, queue, st);
  else if (minb >= 6)
    scan_launch_one<P, MODE, 6>(a, list, cnt, masks, xref, flag, queue, st);
  else
    scan_launch_one<P, MODE, 4>(a, list, cnt, masks, xref, flag, queue, st);
}

template <int P>
void dispatch_scan(bool list_mode, const NbArgs& a, cudaStream_t st) {
  if (!list_mode && a.team) {
    k_rho_team<P, kTeamLanes><<<a.n_tiles * kTeamLanes, a.tile_size, 0, st>>>(
        a.pos, a.start, a.keys, a.tiles, a.scenes, a.wave, a.rho_p, a.nbr_cnt, a.nbm, a.n_total, a.vel, a.pairs,
        a.irho, a.status);
    return;
  }
  if (list_mode)
    scan_variant<P, MODE_LIST>(a.scan_minb, a, a.vlist, a.vcnt, nullptr, a.xref, a.flag, nullptr, st);
  else
    scan_variant<P, MODE_DENSITY>(a.scan_minb, a, nullptr, a.nbr_cnt, a.nbm, nullptr, nullptr,
                                  a.queue, st);
}

template <int P, int MB>
void force_variant(const NbArgs& a, cudaStream_t st) {
  int32_t* queue = a.queue ? a.queue + 1 : nullptr;
  auto kern = queue ? k_force<P, MB, true> : k_force<P, MB, false>;
  int grid = a.n_tiles;
  if (queue) {
    cudaMemsetAsync(queue, 0, sizeof(int32_t), st);
    grid = queue_grid(kern, a.tile_size, a.n_tiles);
  }
  kern<<<grid, a.tile_size, 0, st>>>(a.pos, a.rho_p, a.start, a.keys, a.tiles, a.scenes, a.wave, a.force, a.nbm,
                                     a.nbr_cnt, a.n_total, a.pairs, a.irho, a.status, a.order, queue,
                                     a.n_tiles);
}

template <int P>
void dispatch_force(const NbArgs& a, cudaStream_t st) {
  if constexpr (P == CWA_PREC_COMPENSATED) {
    if (a.team) {
      k_force_team<kTeamLanes><<<a.n_tiles * kTeamLanes, a.tile_size, 0, st>>>(
          a.pos, a.rho_p, a.start, a.keys, a.tiles, a.scenes, a.wave, a.force, a.nbm, a.nbr_cnt, a.n_total,
          a.pairs, a.status);
      return;
    }
  }
  // FP64 keeps eight CTAs a SM for nine: its 56-register form spills more
  if constexpr (P != CWA_PREC_FP64) {
    if (a.force_minb >= 9) {
      force_variant<P, 9>(a, st);
      return;
    }
  }
  if (a.force_minb >= 8)
    force_variant<P, 8>(a, st);
  else
    force_variant<P, 6>(a, st);
}

}  // namespace

cudaError_t launch_scan_cands(int precision, bool list_mode, const NbArgs& a, cudaStream_t stream) {
  if (a.n_tiles <= 0) return cudaSuccess;
  switch (precision) {
    case CWA_PREC_FP32: dispatch_scan<CWA_PREC_FP32>(list_mode, a, stream); break;
    case CWA_PREC_FP64: dispatch_scan<CWA_PREC_FP64>(list_mode, a, stream); break;
    default: dispatch_scan<CWA_PREC_COMPENSATED>(list_mode, a, stream);
  }
  return cudaGetLastError();
}

cudaError_t launch_rho_list(int precision, const NbArgs& a, cudaStream_t stream) {
  if (a.n_tiles <= 0) return cudaSuccess;
#define CWA_RHO_LIST(P)                                                                                     \
  k_rho_list<P><<<a.n_tiles, a.tile_size, 0, stream>>>(a.pos, a.start, a.keys, a.tiles, a.scenes, a.wave,  \
                                                       a.rho_p, a.vlist, a.vcnt, a.nbm, a.nbr_cnt, a.n_total, \
                                                       a.vel, a.pairs, a.irho)
  switch (precision) {
    case CWA_PREC_FP32: CWA_RHO_LIST(CWA_PREC_FP32); break;
    case CWA_PREC_FP64: CWA_RHO_LIST(CWA_PREC_FP64); break;
    default: CWA_RHO_LIST(CWA_PREC_COMPENSATED);
  }
#undef CWA_RHO_LIST
  return cudaGetLastError();
}

cudaError_t launch_force(int precision, const NbArgs& a, cudaStream_t stream) {
  if (a.n_tiles <= 0) return cudaSuccess;
  switch (precision) {
    case CWA_PREC_FP32: dispatch_force<CWA_PREC_FP32>(a, stream); break;
    case CWA_PREC_FP64: dispatch_force<CWA_PREC_FP64>(a, stream); break;
    default: dispatch_force<CWA_PREC_COMPENSATED>(a, stream);
  }
  return cudaGetLastError();
}

}  // namespace cwa
