// cwa_pbd.cu — position-based box collisions on the uniform grid: the
// reference's GridTestPbdGpu3D demo (UniformGrid2D/UniformGridGpu3D.cpp:
// 128-183, 292-346; uniform_grid_pbd_3D_cs.glsl:113-382).
//
// One substep: boxes are inserted into every cell their AABB overlaps
// (COMPUTE_COUNTS / scan / INSERT_BOXES), PreAnimate predicts p = x + dt v,
// the collision query finds each box's contacts with the extents and with
// the boxes of higher index (the home-cell test visits each pair once), and
// PostAnimate applies the averaged displacements with SOR factor k and
// restitution e.
//
// The shader accumulates every contact into both boxes with float atomics,
// so its sums (and the wall terms, added without atomics beside them) depend
// on thread order.  Here the accumulation is a gather: the query writes each
// contact once into the lower box's pair slots and its slot number into a
// list of the higher box, and PostAnimate sums, per box, its wall terms, then
// the pairs it owns in slot order, then the pairs it is the partner of in slot
// order (it sorts its list).  Every float operation is rounded to nearest in
// a fixed order (round-to-nearest intrinsics), so a step is deterministic
// and the float32 CPU restatement reproduces it bit for bit.  Cell ids are
// (i ny + j) nz + k; the shader's (i ny + j) nx + k is the same on its cubic
// grid.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <string>
#include <vector>

#include "cwa_device.cuh"
#include "cwa_internal.h"

namespace cwa {
namespace {

__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fd(float a, float b) { return __fdiv_rn(a, b); }

struct PbdConst {
  int n, nx, ny, nz, maxc, pcap;
  float lo[3], hi[3], cell[3];
  float g[3], dt, damping, k, k_static, sleep, mu_k, mu_s, e;
};

struct PbdPair {
  int32_t i, j;
  float wi, wj;
  float disp[3];
  float frict[3];
};

__device__ __forceinline__ float len3(float x, float y, float z) {
  return __fsqrt_rn(fa(fa(fm(x, x), fm(y, y)), fm(z, z)));
}

__device__ __forceinline__ int cell_c(const PbdConst& c, float p, int a) {
  const int n = a == 0 ? c.nx : (a == 1 ? c.ny : c.nz);
  return cell_axis(p, c.lo[a], c.cell[a], n);
}

__device__ __forceinline__ int cell_id(const PbdConst& c, int i, int j, int k) { return (i * c.ny + j) * c.nz + k; }

// COMPUTE_COUNTS / INSERT_BOXES: item q = box * maxc + t is the box's t-th
// overlapped cell (x-major, z fastest); unused slots get key -1.  One thread
// an item, so a box's cell counters are bumped side by side instead of one
// returned atomic after another.  The box's first thread also clears its
// contact state and runs PreAnimate (:354-370), which touches nothing the
// cells come from.
__global__ void k_pbd_cells(PbdConst c, cwa_pbd_box* __restrict__ boxes, int32_t* __restrict__ ikey,
                            int32_t* __restrict__ islot, int32_t* __restrict__ count, int32_t* __restrict__ rcount,
                            int32_t* status) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= c.n * c.maxc) return;
  const int b = q / c.maxc, t = q - b * c.maxc;
  cwa_pbd_box& o = boxes[b];
  int lo[3], hi[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    lo[a] = cell_c(c, fs(o.x[a], o.hw[a]), a);
    hi[a] = cell_c(c, fa(o.x[a], o.hw[a]), a);
  }
  const int ny = hi[1] - lo[1] + 1, nz = hi[2] - lo[2] + 1, cells = (hi[0] - lo[0] + 1) * ny * nz;
  int key = -1;
  if (t < cells) {
    const int xy = t / nz;
    key = cell_id(c, lo[0] + xy / ny, lo[1] + xy % ny, lo[2] + t - xy * nz);
    islot[q] = count_slot(count, key);
  }
  ikey[q] = key;
  if (t != 0) return;
  if (cells > c.maxc) atomicOr(status, kStatusBigCell);
  rcount[b] = 0;
  float v[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const float ga = a < 3 ? c.g[a] : 0.0f;
    v[a] = fm(c.damping, fa(o.v[a], fm(c.dt, ga)));
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    o.color[a] = 1.0f;  // InsertBox resets the colour
    o.dp_n[a] = 0.0f;
    o.dp_t[a] = 0.0f;
    o.p[a] = fa(o.x[a], fm(c.dt, v[a]));
    o.v[a] = v[a];
  }
  o.n = 0.0f;
}

// Arrival-order insert, then the stable rank (members with a smaller index);
// the sorted list holds the members' boxes.
__global__ void k_pbd_insert(const int32_t* __restrict__ key, const int32_t* __restrict__ slot,
                             const int32_t* __restrict__ start, int32_t* __restrict__ list, int32_t n_items) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n_items || key[q] < 0) return;
  list[start[key[q]] + slot[q]] = q;
}

__global__ void k_pbd_rank(const int32_t* __restrict__ key, const int32_t* __restrict__ start,
                           const int32_t* __restrict__ list, int32_t* __restrict__ sorted, int32_t n_items,
                           int32_t per_box) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n_items || key[q] < 0) return;
  const int b = start[key[q]], e = start[key[q] + 1];
  int rank = 0;
  for (int m = b; m < e; ++m) rank += list[m] < q;
  sorted[b + rank] = q / per_box;
}

// Collide (:293-351) for the ordered pair (i < j); false when they do not overlap.
__device__ bool collide(const PbdConst& c, const cwa_pbd_box& bi, const cwa_pbd_box& bj, const float qmin[3],
                        const float qmax[3], const float bmin[3], const float bmax[3], PbdPair* out) {
  float sz[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) sz[a] = fs(fminf(qmax[a], bmax[a]), fmaxf(qmin[a], bmin[a]));
  int comp = 0;
  if (sz[1] < sz[0] && sz[1] < sz[2]) comp = 1;
  if (sz[2] < sz[0] && sz[2] < sz[1]) comp = 2;
  const float dist = fm(0.5f, sz[comp]);
  if (dist < 0.0f) return false;
  const float eps = 1e-8f;
  float dij[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) dij[a] = fs(bj.p[a], bi.p[a]);
  const float den = fa(len3(dij[0], dij[1], dij[2]), eps);
  float ud[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) ud[a] = fd(dij[a], den);
  const float sg = dij[comp] > 0.0f ? 1.0f : (dij[comp] < 0.0f ? -1.0f : 0.0f);
#pragma unroll
  for (int a = 0; a < 3; ++a) out->disp[a] = 0.0f;
  out->disp[comp] = fm(sg, dist);
  const float rs = fa(bi.rm, bj.rm);
  out->wi = fd(bi.rm, rs);
  out->wj = fd(bj.rm, rs);
  float dp[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) dp[a] = fs(fs(bj.x[a], bj.p[a]), fs(bi.x[a], bi.p[a]));
  const float d = fa(fa(fm(dp[0], ud[0]), fm(dp[1], ud[1])), fm(dp[2], ud[2]));
#pragma unroll
  for (int a = 0; a < 3; ++a) dp[a] = fs(dp[a], fm(d, ud[a]));
  const float mag = len3(dp[0], dp[1], dp[2]);
  float s = 1.0f;
  if (mag < fm(c.mu_s, dist)) s = fminf(1.0f, fd(fm(c.mu_k, dist), mag));
#pragma unroll
  for (int a = 0; a < 3; ++a) out->frict[a] = s == 1.0f ? dp[a] : fm(dp[a], s);
  return true;
}

// CollisionQuery (:225-290) for box i against the boxes of higher index, one
// warp a box.  The cells of a row (ci, cj) are consecutive, so a row's members
// are one range of the sorted list; the lanes fetch the rows' ranges side by
// side and test the members of all rows as one sequence, 32 at a time.  A
// contact's slot is the number of contacts before it in list order, which the
// ballots give.  A contact enters its higher box's list in arrival order.
// Latency bounds it (a member costs two dependent loads): one thread a box
// walked ~100 members in turn on 32 CTAs, 296 us at 4096 boxes; this form
// takes 26 us (both with cold caches).
__global__ void __launch_bounds__(128)
    k_pbd_query(PbdConst c, cwa_pbd_box* __restrict__ boxes, const int32_t* __restrict__ cstart,
                const int32_t* __restrict__ csorted, PbdPair* __restrict__ pairs, int32_t* __restrict__ npairs,
                int32_t* __restrict__ rcount, int64_t* __restrict__ rlist, int32_t* status) {
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= c.n) return;  // whole warps leave together
  const cwa_pbd_box bi = boxes[i];
  float qmin[3], qmax[3];
  int lo[3], hi[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    qmin[a] = fs(bi.p[a], bi.hw[a]);
    qmax[a] = fa(bi.p[a], bi.hw[a]);
    lo[a] = cell_c(c, qmin[a], a);
    hi[a] = cell_c(c, qmax[a], a);
  }
  const float4 red = make_float4(1.0f, 0.0f, 0.0f, 1.0f);
  const int ny = hi[1] - lo[1] + 1, nz = hi[2] - lo[2] + 1, rows = (hi[0] - lo[0] + 1) * ny;
  int t = 0;  // contacts so far (warp-uniform)
  for (int row0 = 0; row0 < rows; row0 += 32) {
    // lane l: row row0 + l, its first cell and its members' range
    const int nrow = min(rows - row0, 32);
    int cell0 = 0, first = 0, len = 0;
    if (lane < nrow) {
      const int x = (row0 + lane) / ny;
      cell0 = cell_id(c, lo[0] + x, lo[1] + row0 + lane - x * ny, lo[2]);
      first = cstart[cell0];
      len = cstart[cell0 + nz] - first;
    }
    int incl = len;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += y;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    for (int m0 = 0; m0 < total; m0 += 32) {
      const int m = m0 + lane;
      int row = 0;  // the member's row: the rows whose ranges end at or before m
      for (int k = 0; k + 1 < nrow; ++k) row += m >= __shfl_sync(0xffffffffu, incl, k);
      const int rc = __shfl_sync(0xffffffffu, cell0, row);
      const int r = m + __shfl_sync(0xffffffffu, first - (incl - len), row);
      bool hit = false;
      int j = 0;
      PbdPair pr;
      if (m < total && (j = csorted[r]) > i) {  // Collide returns for i >= j
        int ck = 0;
        while (r >= cstart[rc + ck + 1]) ++ck;
        const cwa_pbd_box& bj = boxes[j];
        float bmin[3], bmax[3];
        int home[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          bmin[a] = fs(bj.x[a], bj.hw[a]);
          bmax[a] = fa(bj.x[a], bj.hw[a]);
          home[a] = max(lo[a], cell_c(c, bmin[a], a));
        }
        if (cell_id(c, home[0], home[1], home[2]) == rc + ck)
          hit = collide(c, bi, bj, qmin, qmax, bmin, bmax, &pr);
      }
      const unsigned hits = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        const int slot = t + __popc(hits & ((1u << lane) - 1u));
        if (slot < c.pcap) {
          const int64_t q = (int64_t)i * c.pcap + slot;  // n x pcap goes up to 2^34
          pr.i = i;
          pr.j = j;
          pairs[q] = pr;
          const int s = atomicAdd(rcount + j, 1);
          if (s < c.pcap) rlist[(size_t)j * c.pcap + s] = q;  // past pcap: long_partners finds them
        } else {
          atomicOr(status, kStatusBigCell);
        }
        // the same value from every writer
        *reinterpret_cast<float4*>(boxes[i].color) = red;
        *reinterpret_cast<float4*>(boxes[j].color) = red;
      }
      t += __popc(hits);
    }
  }
  if (lane == 0) npairs[i] = min(t, c.pcap);
}

// Wall terms, then the own pairs, then the partner pairs; PostAnimate
// (:372-392).  Eight lanes a box: lane k < 3 sums component k of the normal
// displacement, lane k + 3 that of the friction, lane 6 counts, each in the
// fixed order, so a lane's chain is one addition a pair and the pairs' loads
// are shared by the lanes and run ahead of the sums.  The box's partner list
// is sorted first (each entry's rank is the number of smaller ones), in shared
// memory; boxes of more than kPostList partners, or more than their list holds,
// go to long_partners.  One thread a box took 22 us at 4096 boxes, this
// form 11 us, and the list replaces a counting sort of all pair slots (a key
// pass, a scan and two passes over n pcap slots, 19 us).
constexpr int kPostLanes = 8;
constexpr int kPostThreads = 128;
constexpr int kPostTeams = kPostThreads / kPostLanes;
constexpr int kPostList = 64;
constexpr int kPostWindow = 1 << 17;  // boxes a window of long_partners, a bit each

struct PostShared {
  union {
    struct {
      int64_t in[kPostTeams][kPostList], out[kPostTeams][kPostList];
    };
    uint32_t bits[kPostWindow / 32];
  };
  float val[kPostThreads][6];  // long_partners: the values of up to 128 pairs
  int32_t low[kPostThreads];   // and the pairs' lower boxes
  int32_t warp[kPostThreads / 32], next, is_long[kPostTeams];
};

// Adds the partner pairs of box b, whose team is `mine`, in slot order, that is
// by lower box (a box has one pair at most with another), with the whole block.
// The partners share a cell with b, so they are found among the members of b's
// cells: each marks its bit in a window of box numbers if it has a pair with b,
// and the bits name the pairs in order, 128 at a time.  The members are walked
// once a window.  What it costs is a few loads a member, shared by 128 threads;
// the query's one warp has walked the same members.  With one large box of
// the highest index over n - 1 small ones, 64 slots a box, a step takes 493 us
// at 4096 boxes and 5,076 at 20,000; with the box's team alone walking every
// lower box's pairs it took 3,382 and 43,375, and with partners from a
// counting sort of all pair slots 2,861 and 19,440.
__device__ __forceinline__ float long_partners(const PbdConst& c, int b, const cwa_pbd_box* boxes,
                                            const PbdPair* __restrict__ pairs, const int32_t* __restrict__ npairs,
                                            const int32_t* __restrict__ cstart,
                                            const int32_t* __restrict__ csorted, PostShared& sh, bool mine,
                                            float sum) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int lo[3], hi[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    lo[a] = cell_c(c, fs(boxes[b].x[a], boxes[b].hw[a]), a);
    hi[a] = cell_c(c, fa(boxes[b].x[a], boxes[b].hw[a]), a);
  }
  const int ny = hi[1] - lo[1] + 1, nz = hi[2] - lo[2] + 1, rows = (hi[0] - lo[0] + 1) * ny;
  auto slot_of = [&](int i) {  // box i's pair with b, or -1
    const int m = npairs[i];
    const PbdPair* p = pairs + (size_t)i * c.pcap;
    for (int t = 0; t < m; t += 4) {  // four loads in flight
      int j[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) j[u] = t + u < m ? p[t + u].j : -1;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j[u] == b) return t + u;
    }
    return -1;
  };
  const volatile uint32_t* const bits = sh.bits;  // other warps set bits while a warp looks
  int w0 = 0;  // the window's first box
  while (w0 < b) {
    const int per = min((b - w0 - 1) / (32 * kPostThreads) + 1, kPostWindow / 32 / kPostThreads);  // words a thread
    for (int w = tid; w < per * kPostThreads; w += kPostThreads) sh.bits[w] = 0u;
    if (tid == 0) sh.next = b;
    __syncthreads();
    int next = b;  // the first member past the window
    for (int row = warp; row < rows; row += kPostThreads / 32) {
      const int x = row / ny, cell0 = cell_id(c, lo[0] + x, lo[1] + row - x * ny, lo[2]);
      const int e = cstart[cell0 + nz];
      for (int m = cstart[cell0] + lane; m < e; m += 32) {
        const int i = csorted[m], at = i - w0;
        if (i >= b || at < 0) continue;
        if (at >= kPostWindow) {
          next = min(next, i);
        } else if (!(bits[at >> 5] >> (at & 31) & 1u) && slot_of(i) >= 0) {
          atomicOr(&sh.bits[at >> 5], 1u << (at & 31));
        }
      }
    }
    next = __reduce_min_sync(0xffffffffu, next);
    if (lane == 0) atomicMin(&sh.next, next);
    __syncthreads();
    // each thread's words, and the number of bits before them
    int own = 0;
    for (int w = 0; w < per; ++w) own += __popc(sh.bits[tid * per + w]);
    int incl = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += y;
    }
    if (lane == 31) sh.warp[warp] = incl;
    __syncthreads();
    int first = incl - own, total = 0;
    for (int w = 0; w < kPostThreads / 32; ++w) {
      if (w < warp) first += sh.warp[w];
      total += sh.warp[w];
    }
    for (int r0 = 0; r0 < total; r0 += kPostThreads) {
      if (first < r0 + kPostThreads && first + own > r0) {
        int r = first - r0;
        for (int w = 0; w < per; ++w)
          for (uint32_t m = sh.bits[tid * per + w]; m; m &= m - 1u, ++r)
            if (r >= 0 && r < kPostThreads) sh.low[r] = w0 + 32 * (tid * per + w) + __ffs((int)m) - 1;
      }
      __syncthreads();
      const int n = min(total - r0, kPostThreads);
      if (tid < n) {
        const int i = sh.low[tid];
        const PbdPair& pr = pairs[(size_t)i * c.pcap + slot_of(i)];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          sh.val[tid][a] = fm(pr.wj, pr.disp[a]);
          sh.val[tid][a + 3] = fm(pr.wj, pr.frict[a]);
        }
      }
      __syncthreads();
      if (mine) {
        const int k = tid % kPostLanes;
#pragma unroll 8
        for (int r = 0; r < n; ++r) sum = fa(sum, k < 6 ? sh.val[r][min(k, 5)] : 1.0f);
      }
      __syncthreads();
    }
    w0 = sh.next;
    __syncthreads();
  }
  return sum;
}

__global__ void __launch_bounds__(kPostThreads, 8)
    k_pbd_post(PbdConst c, cwa_pbd_box* __restrict__ boxes, const PbdPair* __restrict__ pairs,
               const int32_t* __restrict__ npairs, const int32_t* __restrict__ rcount,
               const int64_t* __restrict__ rlist, const int32_t* __restrict__ cstart,
               const int32_t* __restrict__ csorted) {
  __shared__ PostShared sh;
  const int k = threadIdx.x % kPostLanes, g = threadIdx.x / kPostLanes;
  const int b0 = blockIdx.x * kPostTeams;
  const bool live = b0 + g < c.n;
  const int b = live ? b0 + g : c.n - 1;  // teams past the end compute the last box and store nothing
  const unsigned team = 0xffu << ((threadIdx.x & 31) - k);
  const cwa_pbd_box o = boxes[b];
  float dpn[3] = {0.0f, 0.0f, 0.0f}, dpt[3] = {0.0f, 0.0f, 0.0f}, nn = 0.0f;
  // collisions with the extents (:230-259), on every lane
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float qmin = fs(o.p[a], o.hw[a]), qmax = fa(o.p[a], o.hw[a]);
    const float ov[2] = {fs(c.lo[a], qmin), fs(qmax, c.hi[a])};
    const float dir[2] = {1.0f, -1.0f};
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      if (!(ov[m] > 0.0f)) continue;
      dpn[a] = fa(dpn[a], fm(fm(dir[m], c.k_static), ov[m]));
      nn = fa(nn, c.k_static);
      float dp[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) dp[q] = q == a ? 0.0f : fs(o.x[q], o.p[q]);
      const float mag = len3(dp[0], dp[1], dp[2]);
      float s = 1.0f;
      if (mag < fm(c.mu_s, ov[m])) s = fminf(1.0f, fd(fm(c.mu_k, ov[m]), mag));
#pragma unroll
      for (int q = 0; q < 3; ++q) dpt[q] = fa(dpt[q], s == 1.0f ? dp[q] : fm(dp[q], s));
    }
  }
  // this lane's component: its sum so far and its value in a pair
  float sum = k < 3 ? (k == 0 ? dpn[0] : k == 1 ? dpn[1] : dpn[2])
                    : k < 6 ? (k == 3 ? dpt[0] : k == 4 ? dpt[1] : dpt[2]) : nn;
  auto add = [&](const PbdPair& pr, bool own) {
    const float w = own ? -pr.wi : pr.wj;
    const float v = reinterpret_cast<const float*>(&pr)[4 + min(k, 5)];  // disp, then frict
    sum = fa(sum, k < 6 ? fm(w, v) : 1.0f);
  };
  const int no = npairs[b];
  const PbdPair* mine = pairs + (size_t)b * c.pcap;
#pragma unroll 4
  for (int t = 0; t < no; ++t) add(mine[t], true);  // b is the lower box
  const int nr = rcount[b];  // b is the higher box
  const bool is_long = live && (nr > kPostList || nr > c.pcap);
  if (nr <= kPostList && nr <= c.pcap) {
    for (int s = k; s < nr; s += kPostLanes) sh.in[g][s] = rlist[(size_t)b * c.pcap + s];
    __syncwarp(team);
    for (int s = k; s < nr; s += kPostLanes) {
      const int64_t q = sh.in[g][s];
      int rank = 0;
      for (int m = 0; m < nr; ++m) rank += sh.in[g][m] < q;
      sh.out[g][rank] = q;
    }
    __syncwarp(team);
#pragma unroll 4
    for (int s = 0; s < nr; ++s) add(pairs[sh.out[g][s]], false);
  }
  if (k == 0) sh.is_long[g] = is_long;
  if (__syncthreads_or(is_long)) {
    for (int q = 0; q < kPostTeams; ++q)
      if (sh.is_long[q]) sum = long_partners(c, b0 + q, boxes, pairs, npairs, cstart, csorted, sh, g == q, sum);
  }
  nn = __shfl_sync(team, sum, 6, kPostLanes);
  const int a = k < 3 ? k : 0;
  const float dn = __shfl_sync(team, sum, a, kPostLanes), dt = __shfl_sync(team, sum, a + 3, kPostLanes);
  const float op = a == 0 ? o.p[0] : a == 1 ? o.p[1] : o.p[2], ox = a == 0 ? o.x[0] : a == 1 ? o.x[1] : o.x[2];
  float p = op, pe = op;
  if (nn > 0.0f) {
    p = fa(p, fd(fm(c.k, fa(dt, dn)), nn));
    pe = fa(pe, fd(fm(c.k, fa(dt, fm(c.e, dn))), nn));
  }
  const float moved = fs(ox, p);
  const bool awake = len3(__shfl_sync(team, moved, 0, kPostLanes), __shfl_sync(team, moved, 1, kPostLanes),
                          __shfl_sync(team, moved, 2, kPostLanes)) > c.sleep;
  if (live && k < 3) {
    cwa_pbd_box& w = boxes[b];
    w.v[a] = fd(fs(pe, ox), c.dt);
    w.dp_n[a] = dn;
    w.dp_t[a] = dt;
    w.p[a] = p;
    if (awake) w.x[a] = p;
    if (a == 0) w.n = nn;
  }
}

constexpr int kB = 128;
inline unsigned nb(long n) { return (unsigned)((n + kB - 1) / kB); }

}  // namespace
}  // namespace cwa

using namespace cwa;

struct cwa_pbd_sim {
  int device = 0;
  cwa_pbd_params prm{};
  PbdConst k{};
  cudaStream_t stream = nullptr;
  cwa_pbd_box* boxes = nullptr;
  int32_t *ikey = nullptr, *islot = nullptr, *ccount = nullptr, *cstart = nullptr, *clist = nullptr,
          *csorted = nullptr;
  PbdPair* pairs = nullptr;
  int32_t *npairs = nullptr, *rcount = nullptr;
  int64_t* rlist = nullptr;  // behind the pairs, in their allocation
  void* ws_cells = nullptr;
  ScanWorkspace scan_cells{};
  int32_t* d_status = nullptr;
  int ncells = 0;
  bool uploaded = false;
  cudaGraphExec_t graph = nullptr;
};

namespace {

cwa_status perr(const std::string& m, cwa_status s = CWA_ERR_INVALID_ARG) {
  cwa::set_error(m);
  return s;
}

#define PBD_CUDA(expr)                                                   \
  do {                                                                   \
    cudaError_t e_ = (expr);                                             \
    if (e_ != cudaSuccess) {                                             \
      cwa::set_error(std::string(#expr) + ": " + cudaGetErrorString(e_)); \
      cudaGetLastError(); /* clear a non-sticky error for the next call */ \
      return e_ == cudaErrorMemoryAllocation ? CWA_ERR_OOM : CWA_ERR_CUDA; \
    }                                                                    \
  } while (0)

void free_items(cwa_pbd_sim* s) {
  cudaFree(s->ikey);  // the four arrays are one allocation
  s->ikey = s->islot = s->clist = s->csorted = nullptr;
}

void free_pbd(cwa_pbd_sim* s) {
  if (!s) return;
  cudaSetDevice(s->device);
  if (s->stream) cudaStreamSynchronize(s->stream);
  if (s->graph) cudaGraphExecDestroy(s->graph);
  free_items(s);
  void* ps[] = {s->boxes, s->ccount, s->cstart, s->pairs, s->npairs, s->rcount, s->ws_cells, s->d_status};
  for (void* p : ps) cudaFree(p);
  if (s->stream) cudaStreamDestroy(s->stream);
  delete s;
}

cwa_status enqueue_substep(cwa_pbd_sim* s) {
  const PbdConst& c = s->k;
  cudaStream_t st = s->stream;
  const long items = (long)c.n * c.maxc;
  k_pbd_cells<<<nb(items), kB, 0, st>>>(c, s->boxes, s->ikey, s->islot, s->ccount, s->rcount, s->d_status);
  PBD_CUDA(cudaGetLastError());
  PBD_CUDA(scan_launch_two_pass(s->ccount, s->cstart, s->ncells, s->ncells + 1, true, s->scan_cells, st, nullptr));
  k_pbd_insert<<<nb(items), kB, 0, st>>>(s->ikey, s->islot, s->cstart, s->clist, (int32_t)items);
  k_pbd_rank<<<nb(items), kB, 0, st>>>(s->ikey, s->cstart, s->clist, s->csorted, (int32_t)items, c.maxc);
  k_pbd_query<<<nb(32l * c.n), kB, 0, st>>>(c, s->boxes, s->cstart, s->csorted, s->pairs, s->npairs, s->rcount,
                                            s->rlist, s->d_status);
  k_pbd_post<<<(unsigned)(((long)c.n * kPostLanes + kPostThreads - 1) / kPostThreads), kPostThreads, 0, st>>>(
      c, s->boxes, s->pairs, s->npairs, s->rcount, s->rlist, s->cstart, s->csorted);
  PBD_CUDA(cudaGetLastError());
  return CWA_OK;
}

cwa_status read_pbd_status(cwa_pbd_sim* s) {
  int32_t v = 0;
  PBD_CUDA(cudaMemcpyAsync(&v, s->d_status, 4, cudaMemcpyDeviceToHost, s->stream));
  PBD_CUDA(cudaStreamSynchronize(s->stream));
  if (v == 0) return CWA_OK;
  PBD_CUDA(cudaMemsetAsync(s->d_status, 0, 4, s->stream));
  PBD_CUDA(cudaStreamSynchronize(s->stream));
  if (v & kStatusNonFinite) return perr("non-finite box position", CWA_ERR_NONFINITE);
  return perr("a box overlapped more cells, or had more contacts, than its slots hold", CWA_ERR_CAPACITY);
}

}  // namespace

extern "C" {

cwa_status cwa_pbd_create(const cwa_pbd_params* p, int32_t device, cwa_pbd_sim** out) {
  if (!p || !out) return perr("null params or output");
  *out = nullptr;
  if (p->n_boxes < 1 || p->n_boxes > (1 << 22)) return perr("n_boxes must be in [1, 2^22]");
  for (int a = 0; a < 3; ++a) {
    if (p->grid_cells[a] < 1 || p->grid_cells[a] > 1024) return perr("grid_cells must be in [1, 1024]");
    if (!(p->extents_hi[a] > p->extents_lo[a])) return perr("extents must have hi > lo");
  }
  if (!(p->dt > 0.0f) || p->substeps < 0) return perr("dt must be positive and substeps >= 0");
  if (p->max_contacts < 0 || p->max_contacts > 4096) return perr("max_contacts must be in [0, 4096]");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
    return perr("no such CUDA device", CWA_ERR_NO_DEVICE);
  cwa_pbd_sim* s = new cwa_pbd_sim();
  s->device = device;
  s->prm = *p;
  PbdConst& k = s->k;
  k.n = p->n_boxes;
  k.nx = p->grid_cells[0];
  k.ny = p->grid_cells[1];
  k.nz = p->grid_cells[2];
  for (int a = 0; a < 3; ++a) {
    k.lo[a] = p->extents_lo[a];
    k.hi[a] = p->extents_hi[a];
    k.cell[a] = (k.hi[a] - k.lo[a]) / (float)p->grid_cells[a];  // mCellSize = extents / cells
    k.g[a] = p->g[a];
  }
  k.dt = p->dt;
  k.damping = p->damping;
  k.k = p->k;
  k.k_static = p->k_static;
  k.sleep = p->sleep_thresh;
  k.mu_k = p->mu_k;
  k.mu_s = p->mu_s;
  k.e = p->e;
  k.maxc = 8;
  k.pcap = p->max_contacts > 0 ? p->max_contacts : 64;
  s->ncells = k.nx * k.ny * k.nz;
  const size_t slots = (size_t)k.n * k.pcap;
  cudaError_t e = cudaSetDevice(device);
  auto al = [&](void** ptr, size_t bytes) {
    if (e == cudaSuccess) e = cudaMalloc(ptr, bytes > 0 ? bytes : 4);
  };
  al((void**)&s->boxes, sizeof(cwa_pbd_box) * k.n);
  al((void**)&s->ccount, 4 * (size_t)s->ncells);
  al((void**)&s->cstart, 4 * ((size_t)s->ncells + 1));
  al((void**)&s->pairs, (sizeof(PbdPair) + sizeof(int64_t)) * slots);
  if (e == cudaSuccess) s->rlist = reinterpret_cast<int64_t*>(s->pairs + slots);
  al((void**)&s->npairs, 4 * (size_t)k.n);
  al((void**)&s->rcount, 4 * (size_t)k.n);
  al(&s->ws_cells, scan_workspace_bytes(s->ncells + 1));
  al((void**)&s->d_status, 4);
  if (e == cudaSuccess) e = cudaMemset(s->ccount, 0, 4 * (size_t)s->ncells);
  if (e == cudaSuccess) e = cudaMemset(s->npairs, 0, 4 * (size_t)k.n);
  if (e == cudaSuccess) e = cudaMemset(s->d_status, 0, 4);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    cwa::set_error(std::string("cwa_pbd_create: ") + cudaGetErrorString(e));
    cudaGetLastError();  // clear a non-sticky error for the next call
    free_pbd(s);
    return e == cudaErrorMemoryAllocation ? CWA_ERR_OOM : CWA_ERR_CUDA;
  }
  scan_bind_workspace(s->ws_cells, s->ncells + 1, &s->scan_cells);
  *out = s;
  return CWA_OK;
}

cwa_status cwa_pbd_destroy(cwa_pbd_sim* s) {
  if (!s) return perr("null sim");
  free_pbd(s);
  return CWA_OK;
}

cwa_status cwa_pbd_upload(cwa_pbd_sim* s, const cwa_pbd_box* host, int32_t n) {
  if (!s) return perr("null sim");
  if (!host || n != s->k.n) return perr("upload size must equal n_boxes");
  PBD_CUDA(cudaSetDevice(s->device));
  // cells a box can overlap: per axis floor(2 hw / cell) + 2, over the largest box
  float hmax[3] = {0.0f, 0.0f, 0.0f};
  for (int i = 0; i < n; ++i)
    for (int a = 0; a < 3; ++a) {
      if (!(host[i].hw[a] >= 0.0f) || !isfinite(host[i].hw[a])) return perr("half widths must be finite, >= 0");
      hmax[a] = std::max(hmax[a], host[i].hw[a]);
    }
  long maxc = 1;
  const int dims[3] = {s->k.nx, s->k.ny, s->k.nz};
  for (int a = 0; a < 3; ++a)
    maxc *= std::min<long>(dims[a], (long)floorf(2.0f * hmax[a] / s->k.cell[a]) + 2);
  if (maxc * n > (1l << 30)) return perr("boxes too large for the grid", CWA_ERR_CAPACITY);
  if (maxc != s->k.maxc || !s->ikey) {
    if (s->graph) {  // it holds the old item buffers
      cudaGraphExecDestroy(s->graph);
      s->graph = nullptr;
    }
    free_items(s);
    s->uploaded = false;  // no step until an upload has its buffers
    s->k.maxc = (int)maxc;
    const size_t items = (size_t)maxc * n;
    PBD_CUDA(cudaMalloc((void**)&s->ikey, 16 * items));
    s->islot = s->ikey + items;
    s->clist = s->islot + items;
    s->csorted = s->clist + items;
  }
  PBD_CUDA(cudaMemcpyAsync(s->boxes, host, sizeof(cwa_pbd_box) * n, cudaMemcpyHostToDevice, s->stream));
  PBD_CUDA(cudaStreamSynchronize(s->stream));
  s->uploaded = true;
  return CWA_OK;
}

cwa_status cwa_pbd_download(cwa_pbd_sim* s, cwa_pbd_box* host, int32_t n) {
  if (!s) return perr("null sim");
  if (!host || n != s->k.n) return perr("download size must equal n_boxes");
  PBD_CUDA(cudaSetDevice(s->device));
  PBD_CUDA(cudaMemcpyAsync(host, s->boxes, sizeof(cwa_pbd_box) * n, cudaMemcpyDeviceToHost, s->stream));
  PBD_CUDA(cudaStreamSynchronize(s->stream));
  return read_pbd_status(s);
}

cwa_status cwa_pbd_step(cwa_pbd_sim* s, int32_t n_steps) {
  if (!s) return perr("null sim");
  if (n_steps < 0) return perr("n_steps < 0");
  if (!s->uploaded) return perr("upload boxes first (cwa_pbd_upload)");
  PBD_CUDA(cudaSetDevice(s->device));
  if (!s->graph && s->prm.substeps > 0) {
    cudaGraph_t g = nullptr;
    PBD_CUDA(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
    cwa_status st = CWA_OK;
    for (int sub = 0; sub < s->prm.substeps && st == CWA_OK; ++sub) st = enqueue_substep(s);
    cudaError_t e = cudaStreamEndCapture(s->stream, &g);
    if (st != CWA_OK) {
      if (g) cudaGraphDestroy(g);
      return st;
    }
    PBD_CUDA(e);
    e = cudaGraphInstantiate(&s->graph, g, 0);
    cudaGraphDestroy(g);
    PBD_CUDA(e);
  }
  for (int32_t k = 0; k < n_steps && s->graph; ++k) PBD_CUDA(cudaGraphLaunch(s->graph, s->stream));
  return CWA_OK;
}

cwa_status cwa_pbd_pair_count(cwa_pbd_sim* s, int64_t* pairs) {
  if (!s || !pairs) return perr("null sim or output");
  PBD_CUDA(cudaSetDevice(s->device));
  std::vector<int32_t> v((size_t)s->k.n);
  PBD_CUDA(cudaMemcpyAsync(v.data(), s->npairs, 4 * v.size(), cudaMemcpyDeviceToHost, s->stream));
  PBD_CUDA(cudaStreamSynchronize(s->stream));
  int64_t total = 0;
  for (const int32_t x : v) total += x;
  *pairs = total;
  return read_pbd_status(s);
}

}  // extern "C"
