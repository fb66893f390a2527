// The MAS-PCG iterations of a small or medium system in one cooperative
// kernel (ys_mas.cu adds it as a body of the solve's conditional node).
//
// A graph of five to seven kernels an iteration costs its launches and the
// tails of grids that are far too small for the chip, where the data of an
// iteration sits in the 126 MB L2.  Here a resident grid (one CTA of 512
// threads an SM, fewer for tiny systems) runs every iteration itself, with
// four grid barriers:
//   A  q = H p, p.q                       | barrier, every CTA sums the partials
//   B  x += alpha p, r -= alpha q, r.r, level-1 residuals      | barrier
//   C  z_d = A_d^-1 r_d for the domains of all levels, r.z     | barrier + sums
//   D  z = sum_l w_l z_l, p = z + beta p                       | barrier
// r.z is summed domain by domain, r.z = sum_l w_l (R_l r).z_l in FP64, so the
// stop test and beta need no pass over z.  Loads that do not wait for a
// barrier's result (row plans, the first tiles of an inverse) are issued
// before it, those that do not wait for the sums before the sums.  Every CTA
// forms the scalars from the same partials in the same order, so all take the
// same decisions; the sums have a fixed order (deterministic).
//
// The wide form, for systems with at most a domain a CTA, applies the FP32
// inverses with FP64 residuals, sums and corrections: the preconditioner is
// then one fixed linear map.  On small ill-conditioned contact systems, where
// the FP32 rounding of r and z was what the iteration fought with, it takes a
// third to a sixth of the iterations (336 against 1862 on 70 vertices with
// stiff friction), and a domain a CTA costs no more than in FP32.
//
// Rows longer than a threshold are split into segments over the warps of the
// whole grid.  Their table is a node of the solve's graph (loop_tables_kernel,
// beside the nodes that form the first residual), so it follows the row plan
// that stands in the caller's buffers at each launch, as every other read of
// the plan does.
//
// The sums are formed by P.blocks virtual CTAs, whatever number of CTAs runs
// them (each takes every gridDim.x-th one).  A solve that has the chip to itself
// runs them all at once; solves in flight on other streams share the chip, a
// part of the SMs each (mas_plan_loop has the sizes), and since no sum
// depends on the grid a solution has the same bits either way.
//
// Barrier waits are bounded (kPollLimitParam polls): a CTA that gives up marks
// the solve void (kBarrierFail) and every CTA leaves.
#pragma once

#include "ys_mas.cuh"
#include "ys_mas_dev.cuh"
#include "ys_pcg.cuh"

namespace ys {

constexpr int kLoopThreads = 512;
constexpr uint32_t kLoopCoarse = 512;    // most nodes of the levels from 2 on (their residuals in shared memory)
constexpr uint32_t kLongRow = 64;        // longer rows are split over warps, in segments of twice that
constexpr uint32_t kLoopGroup = 12;      // more level-2 domains than this go three to a CTA
constexpr int kLoopMaxDofs = 4;          // 3-DoF entries a lane holds of a domain of at most 128 DoF

// What the loop needs to know of the row plan and of the domains; written by
// loop_tables_kernel at every launch.
struct LoopTable {
  uint32_t threshold;      // longer rows (per block set) are split
  uint32_t num_segments, num_long;
  uint32_t level_domain[kMaxLevels + 1];  // first domain of each level
};

struct LoopParams {
  SpmvSet sets[2];
  int nsets;
  MasDev M;
  double* x;
  double* r;
  double* p;
  float4* p32;
  double* q;
  double* st;
  double* partials;
  unsigned long long* arrivals;
  uint32_t blocks;         // virtual CTAs: every sum is split among these
  int stop_rule;
  uint32_t gemv_warps;     // warps of a CTA with a GEMV area in shared memory
  uint32_t area;           // float4 of one area
  // long rows: segments (row, first entry, last entry, set) ordered by row and
  // set; long_row lists the rows, long_first their first segments
  LoopTable* table;
  uint4* segments;
  uint32_t* long_row;
  uint32_t* long_first;
  uint32_t max_segments;   // room in segments, long_row and seg
  double* seg;             // 3 per segment
  double* zl64;            // the wide form's FP64 level corrections, 3 per packed node
};

// Values other CTAs write in this kernel are read by plain loads (never the
// read-only path); the barrier's acquire makes them current.
__device__ __forceinline__ void loop_x(const float4* x, uint32_t j, float (&v)[3]) {
  const float4 t = x[j];
  v[0] = t.x; v[1] = t.y; v[2] = t.z;
}
__device__ __forceinline__ void loop_x(const double* x, uint32_t j, double (&v)[3]) {
  v[0] = x[3ull * j]; v[1] = x[3ull * j + 1]; v[2] = x[3ull * j + 2];
}

template <typename T>
struct LoopTypes;
template <>
struct LoopTypes<float> {
  using X = float4;
};
template <>
struct LoopTypes<double> {
  using X = double;
};

__device__ __forceinline__ const float* set_values(const SpmvSet& s, float) { return s.values32; }
__device__ __forceinline__ const double* set_values(const SpmvSet& s, double) { return s.values; }

// State of the iteration, the same in every CTA; thread 0 writes it, the
// others read it after the next CTA barrier.
struct LoopState {
  double delta, prev, rr, curv, alpha, beta, it;
  unsigned long long target;
  int status, ok;
  LoopTable t;
};

// Bounded grid barrier on a monotonic arrival count; false: gave up.
__device__ __forceinline__ bool loop_barrier(const LoopParams& P, LoopState& S) {
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned long long target = S.target + gridDim.x;
    S.target = target;
    int good = 1;
    unsigned long long c;
    // release: the CTA's writes (ordered before by the barrier above) are
    // visible to whoever sees the arrival
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(P.arrivals) : "memory");
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(P.arrivals) : "memory");
    if (c < target) {
      const double limit = P.st[kPollLimitParam];
      double polls = 0.0;
      volatile double* fail = P.st + kBarrierFail;
      while (c < target) {
        if (polls >= limit || (((uint32_t)polls & 63u) == 63u && *fail != 0.0)) {
          good = 0;
          *fail = 1.0;
          break;
        }
        polls += 1.0;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(P.arrivals) : "memory");
      }
    }
    S.ok = good;
  }
  __syncthreads();
  return S.ok != 0;
}

// Total of the grid's partials, by every warp for itself (all lanes get it, the
// same bits in every warp and CTA): no CTA barrier on the path.
__device__ __forceinline__ double loop_total(const double* partials, uint32_t blocks) {
  double a = 0.0;
  for (uint32_t b = threadIdx.x & 31; b < blocks; b += 32) a += partials[b];
  return warp_sum(a);
}

// A virtual CTA's sum, in two parts: every warp leaves its own in row k of
// `parts` (k counts the CTA's virtual ones), and once all are there a warp a
// virtual CTA adds the rows.  Nothing waits between the virtual CTAs.
constexpr int kLoopWarps = kLoopThreads / 32;
__device__ __forceinline__ void loop_part(double* parts, int k, double v) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) parts[k * kLoopWarps + (threadIdx.x >> 5)] = v;
}
template <bool SHARED>
__device__ __forceinline__ void loop_parts_end(uint32_t blocks, const double* parts, double* partials) {
  const uint32_t lane = threadIdx.x & 31, k = threadIdx.x >> 5, vb = blockIdx.x + k * gridDim.x;
  __syncthreads();
  if (k < (SHARED ? kLoopShares : 1) && vb < blocks) {
    const double t = warp_sum(lane < kLoopWarps ? parts[k * kLoopWarps + lane] : 0.0);
    if (lane == 0) partials[vb] = t;
  }
}

// The long rows' segments, a warp each; returns the lane's share of p.q.
template <typename T>
__device__ __forceinline__ double loop_segments(const LoopParams& P, const LoopState& L,
                                                const typename LoopTypes<T>::X* px, uint32_t vb, uint32_t blocks) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double dot = 0.0;
  for (uint32_t s = warp * blocks + vb; s < L.t.num_segments; s += kLoopWarps * blocks) {
    const uint4 it = __ldg(P.segments + s);
    const SpmvSet& S = P.sets[it.w];
    const T* vals = set_values(S, T(0));
    T a0 = 0, a1 = 0, a2 = 0;
#pragma unroll 2
    for (uint32_t e = it.y + lane; e < it.z; e += 32) {
      const uint32_t eb = __ldg(S.entry_block + e), j = __ldg(S.entry_col + e);
      T b[9], xv[3];
      loop_x(px, j, xv);
      load_block(vals, eb & 0x7fffffffu, b);
      block_mac(b, xv, (eb & 0x80000000u) != 0, a0, a1, a2);
    }
    a0 = warp_sum(a0);
    a1 = warp_sum(a1);
    a2 = warp_sum(a2);
    if (lane == 0) {
      P.seg[3ull * s] = (double)a0;
      P.seg[3ull * s + 1] = (double)a1;
      P.seg[3ull * s + 2] = (double)a2;
      const double* p = P.p + 3ull * it.x;
      dot += p[0] * (double)a0 + p[1] * (double)a1 + p[2] * (double)a2;
    }
  }
  return dot;
}

// Eight lanes a row, U rows a group of lanes at a time (rows of the CTA's
// contiguous range, so neighbours meet in L1), two entries a lane and row in
// flight.  The row bounds and the first two entries' indices of a round are
// loaded a round ahead (those of the first before the barrier that completes
// p): what is left on the path from the barrier is the gather of p.
template <typename T, int U>
struct LoopRows {
  uint32_t e0[U], e1[U];
  uint32_t eb[U][2], col[U][2];

  __device__ __forceinline__ void bounds(const LoopParams& P, const LoopState& L, uint32_t base,
                                         uint32_t r1) {
    const SpmvSet& S = P.sets[0];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t i = base + u * (kLoopThreads / 8);
      const bool valid = i < r1;
      e0[u] = valid ? __ldg(S.row_ptr + i) : 0u;
      e1[u] = valid ? __ldg(S.row_ptr + i + 1) : 0u;
      if (e1[u] - e0[u] > L.t.threshold) e1[u] = e0[u];
    }
  }
  __device__ __forceinline__ void indices(const LoopParams& P, int sub) {
    const SpmvSet& S = P.sets[0];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const uint32_t e = e0[u] + sub + kRowLanes * m;
        const uint32_t k = e < e1[u] ? e : 0u;  // entry 0 stands in (its product is dropped)
        eb[u][m] = __ldg(S.entry_block + k);
        col[u][m] = __ldg(S.entry_col + k);
      }
  }
};

// q = H p for this CTA's rows over one block set; returns the thread's share
// of p.q.  R holds the first round's rows on entry and those from `next` on
// exit.
template <typename T, int U>
__device__ __forceinline__ double loop_spmv(const LoopParams& P, const LoopState& L,
                                            const typename LoopTypes<T>::X* px, LoopRows<T, U>& R, uint32_t first,
                                            uint32_t r1, uint32_t next, uint32_t next_r1) {
  constexpr uint32_t kRows = kLoopThreads / 8;
  const int sub = threadIdx.x & 7;
  const SpmvSet& S = P.sets[0];
  const T* vals = set_values(S, T(0));
  double dot = 0.0;
  // every lane runs the same rounds (the shuffles need whole warps)
  const uint32_t warp_first = first - ((threadIdx.x & 31) >> 3);
  for (uint32_t wb = warp_first; wb < r1; wb += U * kRows) {
    const uint32_t base = wb + ((threadIdx.x & 31) >> 3);
    T a[U][3];
    uint32_t e0[U], e1[U];
    double pr[U][3];
    {
      T xv[U][2][3], b[U][2][9];
      uint32_t tr[U][2];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          loop_x(px, R.col[u][m], xv[u][m]);
          load_block(vals, R.eb[u][m] & 0x7fffffffu, b[u][m]);
          tr[u][m] = R.eb[u][m] & 0x80000000u;
        }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        e0[u] = R.e0[u];
        e1[u] = R.e1[u];
        const uint32_t i = base + u * kRows;
        if (i < r1 && sub == 0)
#pragma unroll
          for (int k = 0; k < 3; ++k) pr[u][k] = P.p[3ull * i + k];
      }
      // the next round's rows (those from `next` after the last)
      const bool more = wb + U * kRows < r1;
      R.bounds(P, L, more ? base + U * kRows : next, more ? r1 : next_r1);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        a[u][0] = a[u][1] = a[u][2] = 0;
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          T t0 = a[u][0], t1 = a[u][1], t2 = a[u][2];
          block_mac(b[u][m], xv[u][m], tr[u][m] != 0, t0, t1, t2);
          if (e0[u] + sub + kRowLanes * m < e1[u]) {
            a[u][0] = t0;
            a[u][1] = t1;
            a[u][2] = t2;
          }
        }
      }
    }
    R.indices(P, sub);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      for (uint32_t e = e0[u] + sub + 2 * kRowLanes; e < e1[u]; e += kRowLanes) {
        const uint32_t eb = __ldg(S.entry_block + e), j = __ldg(S.entry_col + e);
        T b[9], xv[3];
        loop_x(px, j, xv);
        load_block(vals, eb & 0x7fffffffu, b);
        block_mac(b, xv, (eb & 0x80000000u) != 0, a[u][0], a[u][1], a[u][2]);
      }
#pragma unroll
      for (int o = kRowLanes / 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 3; ++k) a[u][k] += __shfl_xor_sync(0xffffffffu, a[u][k], o, kRowLanes);
      const uint32_t i = base + u * kRows;
      if (i < r1 && sub == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          P.q[3ull * i + k] = (double)a[u][k];
          dot += pr[u][k] * (double)a[u][k];
        }
      }
    }
  }
  return dot;
}

// The same over two block sets (a static and a dynamic one), a row at a time.
template <typename T>
__device__ __forceinline__ double loop_spmv_sets(const LoopParams& P, const LoopState& L,
                                                 const typename LoopTypes<T>::X* px, uint32_t first, uint32_t r1) {
  const int sub = threadIdx.x & 7;
  double dot = 0.0;
  const uint32_t in_warp = (threadIdx.x & 31) >> 3;
  for (uint32_t wb = first - in_warp; wb < r1; wb += kLoopThreads / 8) {
    const uint32_t i = wb + in_warp;
    const bool valid = i < r1;
    double q[3] = {0.0, 0.0, 0.0};
    for (int s = 0; s < P.nsets; ++s) {
      const SpmvSet& S = P.sets[s];
      const T* vals = set_values(S, T(0));
      const uint32_t e0 = valid ? __ldg(S.row_ptr + i) : 0u, end = valid ? __ldg(S.row_ptr + i + 1) : 0u;
      const uint32_t e1 = end - e0 > L.t.threshold ? e0 : end;
      T a[3] = {0, 0, 0};
      for (uint32_t e = e0 + sub; e < e1; e += kRowLanes) {
        const uint32_t eb = __ldg(S.entry_block + e), j = __ldg(S.entry_col + e);
        T b[9], xv[3];
        loop_x(px, j, xv);
        load_block(vals, eb & 0x7fffffffu, b);
        block_mac(b, xv, (eb & 0x80000000u) != 0, a[0], a[1], a[2]);
      }
#pragma unroll
      for (int o = kRowLanes / 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 3; ++k) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o, kRowLanes);
#pragma unroll
      for (int k = 0; k < 3; ++k) q[k] += (double)a[k];
    }
    if (valid && sub == 0) {
      const double* p = P.p + 3ull * i;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        P.q[3ull * i + k] = q[k];
        dot += p[k] * q[k];
      }
    }
  }
  return dot;
}

// x += alpha p, r -= alpha q for a fine variable, in two parts: the loads do
// not wait for alpha.
struct LoopUpdate {
  double q[3], p[3], x[3], r[3];
  __device__ __forceinline__ void load(const LoopParams& P, const LoopState& L, uint32_t i) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      q[k] = P.q[3ull * i + k];
      p[k] = P.p[3ull * i + k];
      x[k] = P.x[3ull * i + k];
      r[k] = P.r[3ull * i + k];
    }
    if (L.t.num_long) {
      bool is_long = false;
      for (int s = 0; s < P.nsets; ++s)
        is_long |= __ldg(P.sets[s].row_ptr + i + 1) - __ldg(P.sets[s].row_ptr + i) > L.t.threshold;
      if (is_long) {
        uint32_t lo = 0, hi = L.t.num_long;  // long_row is ascending
        while (hi - lo > 1) {
          const uint32_t mid = (lo + hi) / 2;
          if (__ldg(P.long_row + mid) <= i) lo = mid;
          else hi = mid;
        }
        for (uint32_t s = __ldg(P.long_first + lo); s < __ldg(P.long_first + lo + 1); ++s)
#pragma unroll
          for (int k = 0; k < 3; ++k) q[k] += P.seg[3ull * s + k];
      }
    }
  }
  // the new residual is left in r; returns its squared norm
  __device__ __forceinline__ double store(const LoopParams& P, uint32_t i, double alpha) {
    double rr = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      P.x[3ull * i + k] = x[k] + p[k] * alpha;
      r[k] = r[k] - q[k] * alpha;
      P.r[3ull * i + k] = r[k];
      rr += r[k] * r[k];
    }
    return rr;
  }
};

// Residual sum of node p (packed id) over its children, by one warp (all
// lanes get it); src holds the children's FP64 residuals, indexed by packed id
// minus src_base.
__device__ __forceinline__ void loop_child_sum(const MasDev& M, uint32_t p, const double* src, uint32_t src_base,
                                               int lane, double (&s)[3]) {
  const uint32_t c = p - M.nv;
  s[0] = s[1] = s[2] = 0.0;
  const uint32_t end = __ldg(M.child_ptr + c + 1);
  for (uint32_t q = __ldg(M.child_ptr + c) + lane; q < end; q += 32) {
    const double* v = src + 3ull * (__ldg(M.child_fine + q) - src_base);
    s[0] += v[0];
    s[1] += v[1];
    s[2] += v[2];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) s[k] = warp_sum(s[k]);
}

// Tiles of a domain's inverse a lane has in flight (3 and 4 spilled registers:
// 27 and 29 us an iteration at 31,744 variables against 24).
constexpr int kLoopTiles = 2;

struct LoopTilesAhead {
  float4 t[kLoopTiles][4];
  __device__ __forceinline__ void load(const float4* src, int k, uint32_t slot, uint32_t tiles) {
    if (slot < tiles) {
#pragma unroll
      for (int m = 0; m < 4; ++m) t[k][m] = __ldg(src + 4ull * slot + m);
    }
  }
  // the first tiles of domain d (they do not wait for the residual)
  __device__ __forceinline__ void first(const MasDev& M, uint32_t d) {
    const uint32_t T = inv_tiles(3 * (__ldg(M.dom_node_ptr + d + 1) - __ldg(M.dom_node_ptr + d)));
    const float4* src = reinterpret_cast<const float4*>(M.inverse + __ldg(M.inv_offset + d));
#pragma unroll
    for (int k = 0; k < kLoopTiles; ++k) load(src, k, (threadIdx.x & 31) + 32 * k, T * (T + 1) / 2);
  }
};

// z_d = A_d^-1 r_d by one warp from its area of shared memory; `ahead` holds
// the domain's first tiles, res the FP64 residuals of its level, indexed by
// packed id minus res_base.  Returns the lane's share of w r_d . z_d.
__device__ __forceinline__ double loop_gemv(const LoopParams& P, uint32_t d, LoopTilesAhead& ahead, const double* res,
                                            uint32_t res_base, double w, float4* area) {
  const MasDev& M = P.M;
  const int lane = threadIdx.x & 31;
  const uint32_t nb = __ldg(M.dom_node_ptr + d), n = 3 * (__ldg(M.dom_node_ptr + d + 1) - nb);
  const uint32_t T = inv_tiles(n), ld = gemv_partial_ld(T), tiles = T * (T + 1) / 2;
  const float4* src = reinterpret_cast<const float4*>(M.inverse + __ldg(M.inv_offset + d));
  float4* part = area;
  float* rloc = reinterpret_cast<float*>(area + T * ld);
  double rv[kLoopMaxDofs];
  uint32_t node[kLoopMaxDofs];
#pragma unroll
  for (int k = 0; k < kLoopMaxDofs; ++k) {
    const uint32_t t = lane + 32 * k;
    rv[k] = 0.0;
    node[k] = 0;
    if (t < n) {
      node[k] = __ldg(M.dom_nodes + nb + t / 3);
      rv[k] = res[3ull * (node[k] - res_base) + t % 3];
    }
    if (t < 4 * T) rloc[t] = (float)rv[k];
  }
  __syncwarp();
  const float4* r4 = reinterpret_cast<const float4*>(rloc);
  for (uint32_t s0 = lane; s0 < tiles; s0 += 32 * kLoopTiles) {
#pragma unroll
    for (int k = 0; k < kLoopTiles; ++k) {
      const uint32_t slot = s0 + 32 * k;
      if (slot < tiles) gemv_tile(T, ld, slot, ahead.t[k], r4, part);
      ahead.load(src, k, slot + 32 * kLoopTiles, tiles);
    }
  }
  __syncwarp();
  double dot = 0.0;
#pragma unroll
  for (int k = 0; k < kLoopMaxDofs; ++k) {
    const uint32_t i = lane + 32 * k;
    if (i >= n) continue;
    const float* row = reinterpret_cast<const float*>(part + (i / 4) * ld) + (i % 4);
    float s0 = 0.0f, s1 = 0.0f;
    for (uint32_t y = 0; y < T; y += 2) {  // T is even
      s0 += row[4 * y];
      s1 += row[4 * y + 4];
    }
    const float z = s0 + s1;
    M.zl[3ull * node[k] + i % 3] = z;
    dot += rv[k] * (double)z;
  }
  __syncwarp();
  return w * dot;
}

// A tile's products in the CTA form: the same cells as gemv_tile, R the type
// of the residual and of the sums.
template <typename R>
struct alignas(16) Quad {
  R v[4];
};
template <typename R>
__device__ __forceinline__ void loop_tile(uint32_t T, uint32_t ld, uint32_t slot, const float4 (&t)[4], const R* r,
                                          Quad<R>* part) {
  // see gemv_tile for the slot's (A, B)
  const uint32_t q = (uint32_t)(((float)slot + 0.5f) * (1.0f / (float)(T + 1)));
  const uint32_t c = slot - q * (T + 1);
  const bool first = c < T - q;
  const uint32_t A = first ? q : T - 1 - q;
  const uint32_t B = first ? q + c : A + (c - (T - q));
  const R m[4][4] = {{t[0].x, t[0].y, t[0].z, t[0].w},
                     {t[1].x, t[1].y, t[1].z, t[1].w},
                     {t[2].x, t[2].y, t[2].z, t[2].w},
                     {t[3].x, t[3].y, t[3].z, t[3].w}};
  Quad<R> x = *reinterpret_cast<const Quad<R>*>(r + 4 * B), u;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    u.v[i] = mac(m[i][3], x.v[3], mac(m[i][2], x.v[2], mac(m[i][1], x.v[1], m[i][0] * x.v[0])));
  part[A * ld + B] = u;
  if (A != B) {
    x = *reinterpret_cast<const Quad<R>*>(r + 4 * A);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      u.v[i] = mac(m[3][i], x.v[3], mac(m[2][i], x.v[2], mac(m[1][i], x.v[1], m[0][i] * x.v[0])));
    part[B * ld + A] = u;
  }
}

// z_d = A_d^-1 r_d by the whole CTA, a tile a thread, the tiles prefetched
// before the residuals are summed.
template <typename R>
__device__ __forceinline__ double loop_gemv_cta(const LoopParams& P, uint32_t d, const float4 (&tile)[4],
                                                const double* res, uint32_t res_base, double w, float4* area, R* zl) {
  const MasDev& M = P.M;
  const uint32_t nb = __ldg(M.dom_node_ptr + d), n = 3 * (__ldg(M.dom_node_ptr + d + 1) - nb);
  const uint32_t T = inv_tiles(n), ld = gemv_partial_ld(T), tiles = T * (T + 1) / 2;
  Quad<R>* part = reinterpret_cast<Quad<R>*>(area);
  R* rloc = reinterpret_cast<R*>(part + T * ld);
  const uint32_t t = threadIdx.x;
  double rv = 0.0;
  uint32_t node = 0;
  if (t < n) {
    node = __ldg(M.dom_nodes + nb + t / 3);
    rv = res[3ull * (node - res_base) + t % 3];
  }
  if (t < 4 * T) rloc[t] = (R)rv;
  __syncthreads();
  if (t < tiles) loop_tile<R>(T, ld, t, tile, rloc, part);
  const float4* src = reinterpret_cast<const float4*>(M.inverse + __ldg(M.inv_offset + d));
  for (uint32_t slot = t + kLoopThreads; slot < tiles; slot += kLoopThreads) {
    float4 more[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) more[m] = __ldg(src + 4ull * slot + m);
    loop_tile<R>(T, ld, slot, more, rloc, part);
  }
  __syncthreads();
  double dot = 0.0;
  if (t < n) {
    const R* row = reinterpret_cast<const R*>(part + (t / 4) * ld) + (t % 4);
    R s0 = 0, s1 = 0;
    for (uint32_t y = 0; y < T; y += 2) {  // T is even
      s0 += row[4 * y];
      s1 += row[4 * y + 4];
    }
    const R z = s0 + s1;
    zl[3ull * node + t % 3] = z;
    dot = w * rv * (double)z;
  }
  __syncthreads();
  return dot;
}

__device__ __forceinline__ void loop_prefetch(const MasDev& M, uint32_t d, float4 (&tile)[4]) {
  const uint32_t T = inv_tiles(3 * (__ldg(M.dom_node_ptr + d + 1) - __ldg(M.dom_node_ptr + d)));
  if (threadIdx.x < T * (T + 1) / 2) {
    const float4* src = reinterpret_cast<const float4*>(M.inverse + __ldg(M.inv_offset + d)) + 4ull * threadIdx.x;
#pragma unroll
    for (int m = 0; m < 4; ++m) tile[m] = __ldg(src + m);
  }
}

// Residuals of the levels 2 .. l that domain d of level l needs, in `coarse`
// (indexed by packed id minus the level-2 offset).
__device__ __forceinline__ void loop_coarse(const LoopParams& P, uint32_t d, uint32_t l, double* coarse) {
  const MasDev& M = P.M;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t l2 = M.level_node_offset[2];
  const uint32_t nb = __ldg(M.dom_node_ptr + d), nn = __ldg(M.dom_node_ptr + d + 1) - nb;
  for (uint32_t lev = 2; lev <= l; ++lev) {
    const uint32_t base = M.level_node_offset[lev];
    const uint32_t count = lev == l ? nn : M.level_node_offset[lev + 1] - base;
    for (uint32_t c = warp; c < count; c += kLoopThreads / 32) {
      const uint32_t p = lev == l ? __ldg(M.dom_nodes + nb + c) : base + c;
      double s[3];
      if (lev == 2) loop_child_sum(M, p, M.rl64, 0u, lane, s);
      else loop_child_sum(M, p, coarse, l2, lane, s);
      if (lane < 3) coarse[3 * (p - l2) + lane] = lane == 0 ? s[0] : (lane == 1 ? s[1] : s[2]);
    }
    __syncthreads();
  }
}

// z_i = sum_l w_l z_l(map_l(i)).
template <bool WIDE>
__device__ __forceinline__ void loop_collect(const LoopParams& P, uint32_t i, double (&z)[3]) {
  if constexpr (!WIDE) {
    collect_levels(P.M, P.M.nv, i, z);
  } else {
    z[0] = z[1] = z[2] = 0.0;
    for (uint32_t l = 0; l < P.M.levels; ++l) {
      const double* v = P.zl64 + 3ull * __ldg(P.M.cmap + (uint64_t)l * P.M.nv + i);
      const double w = (double)P.M.weight[l];
#pragma unroll
      for (int k = 0; k < 3; ++k) z[k] += w * v[k];
    }
  }
}

// SHARED: fewer CTAs than virtual ones (the other form is spared the loops over
// them, and their registers: solve of a 33^3 cube in FP64 1702 -> 1655 us).
template <typename T, bool WIDE, bool SHARED>
__global__ void __launch_bounds__(kLoopThreads, 1) mas_pcg_loop(const __grid_constant__ LoopParams P) {
  extern __shared__ float4 loop_areas[];
  __shared__ double parts[kLoopShares * kLoopWarps];
  __shared__ double coarse[3 * kLoopCoarse];
  __shared__ LoopState S;
  const MasDev& M = P.M;
  double* const st = P.st;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t blocks = SHARED ? P.blocks : gridDim.x;
  const typename LoopTypes<T>::X* px;
  if constexpr (sizeof(T) == 4) px = P.p32;
  else px = P.p;
  if (threadIdx.x == 0) {
    S.delta = st[kDeltaNew];
    S.prev = S.delta;
    S.rr = st[kRR];
    S.it = st[kIter];
    S.curv = S.alpha = S.beta = 0.0;
    S.target = 0ull;
    S.status = (int)st[kStatus];
    S.t = *P.table;
  }
  __syncthreads();
  // rows of a virtual CTA
  const uint32_t per = ((M.nv + blocks - 1) / blocks + 3u) & ~3u;
  auto rows_end = [&](uint32_t vb) { return min(M.nv, (vb + 1) * per); };
  auto rows_begin = [&](uint32_t vb) { return vb * per + (threadIdx.x >> 3); };
  constexpr int U = 1;  // 2 spilled registers: slower
  LoopRows<T, U> rows;
  if (P.nsets == 1) {
    rows.bounds(P, S, rows_begin(blockIdx.x), rows_end(blockIdx.x));
    rows.indices(P, threadIdx.x & 7);
  }
  __syncthreads();
  while (S.status == kContinue) {
    // A
    int k = 0;  // counts the CTA's virtual ones
    for (uint32_t vb = blockIdx.x; vb < blocks; vb += gridDim.x, ++k) {
      const uint32_t first_row = rows_begin(vb), r1 = rows_end(vb);
      double dot;
      if (P.nsets == 1) {
        // what the warp multiplies next: its rows of the CTA's next virtual
        // CTA, or of the first one where that one has none for it
        uint32_t nb = vb;
        if constexpr (SHARED) nb += gridDim.x;
        if (nb >= blocks || nb * per + 4u * warp >= M.nv) nb = blockIdx.x;
        dot = loop_spmv<T, U>(P, S, px, rows, first_row, r1, rows_begin(nb), rows_end(nb));
      } else {
        dot = loop_spmv_sets<T>(P, S, px, first_row, r1);
      }
      if (S.t.num_segments) dot += loop_segments<T>(P, S, px, vb, blocks);
      loop_part(parts, k, dot);
      if constexpr (!SHARED) break;
    }
    loop_parts_end<SHARED>(blocks, parts, P.partials);
    if (!loop_barrier(P, S)) break;
    // the first variables of B are on their way while the step length is summed
    LoopUpdate up;
    uint32_t up_i = 0, up_p = 0, up_q = 0, up_end = 0;
    bool up_on = false;
    auto up_node = [&](uint32_t p) {  // the children of level-1 node p
      up_p = p;
      up_on = false;
      if (p < M.level_node_offset[2]) {
        up_end = __ldg(M.child_ptr + (p - M.nv) + 1);
        up_q = __ldg(M.child_ptr + (p - M.nv)) + lane;
        up_on = up_q < up_end;
        if (up_on) up_i = __ldg(M.child_fine + up_q);
      }
    };
    auto up_first = [&](uint32_t vb) {
      if (M.levels > 1) {
        up_node(M.level_node_offset[1] + warp * blocks + vb);
      } else {
        up_i = vb * kLoopThreads + threadIdx.x;
        up_on = up_i < M.nv;
      }
      if (up_on) up.load(P, S, up_i);
    };
    up_first(blockIdx.x);
    const double curv = loop_total(P.partials, blocks), prev = S.delta;
    const bool restart = isfinite(curv) && curv <= 0.0 && isfinite(prev) && prev > 0.0;
    if (!restart && (!isfinite(curv) || curv <= 0.0)) {
      if (threadIdx.x == 0) {
        S.curv = curv;
        S.alpha = 0.0;
        S.prev = prev;
        S.it += 1.0;
        S.status = kNonSpd;
      }
      break;
    }
    // (restart: finite non-positive curvature, zero step; see spmv_dot_finish)
    const double alpha = restart ? 0.0 : prev / curv;
    // B
    k = 0;
    for (uint32_t vb = blockIdx.x; vb < blocks; vb += gridDim.x, ++k) {
      double acc = 0.0;
      if (M.levels > 1) {
        while (up_p < M.level_node_offset[2]) {  // warp-uniform
          double s[3] = {0.0, 0.0, 0.0};
          while (up_on) {
            acc += up.store(P, up_i, alpha);
#pragma unroll
            for (int k = 0; k < 3; ++k) s[k] += up.r[k];
            up_q += 32;
            up_on = up_q < up_end;
            if (up_on) {
              up_i = __ldg(M.child_fine + up_q);
              up.load(P, S, up_i);
            }
          }
#pragma unroll
          for (int k = 0; k < 3; ++k) s[k] = warp_sum(s[k]);
          if (lane < 3) M.rl64[3ull * up_p + lane] = lane == 0 ? s[0] : (lane == 1 ? s[1] : s[2]);
          up_node(up_p + kLoopWarps * blocks);
          if (up_on) up.load(P, S, up_i);
        }
      } else {
        while (up_on) {
          acc += up.store(P, up_i, alpha);
          up_i += blocks * kLoopThreads;
          up_on = up_i < M.nv;
          if (up_on) up.load(P, S, up_i);
        }
      }
      loop_part(parts, k, acc);
      if constexpr (SHARED) {
        if (vb + gridDim.x < blocks) up_first(vb + gridDim.x);
      }
      if constexpr (!SHARED) break;
    }
    loop_parts_end<SHARED>(blocks, parts, P.partials + 2 * blocks);
    // the first tiles of the warp's (or CTA's) first domain are on their way
    // over the barrier; the coarsest domains go to the first virtual CTAs
    const uint32_t first2 = M.levels > 2 ? S.t.level_domain[2] : M.num_domains;
    const uint32_t first1 = M.levels > 1 ? S.t.level_domain[1] : M.num_domains, n1 = first2 - first1;
    const uint32_t whole = WIDE ? M.num_domains : M.num_domains - first2;  // domains by whole CTAs, from the last
    // of those, a CTA takes one of the levels >= 3 (their residuals are a chain
    // of sums) and one of level 2, or three of many, which leaves more CTAs to
    // the fine levels where a few would only wait for one another.  Apart /
    // three to a CTA, us an iteration in FP32 (FP64) on cloths with bodies:
    // 26.1 / 27.5 (30.4 / 31.9) with 8 level-2 domains, 28.1 / 29.1 (33.9 / 34.9)
    // with 10, 24.1 / 26.5 (27.6 / 29.9) with 11, 37.6 / 33.3 (46.9 / 42.2) with 18,
    // 51.7 / 52.0 (61.5 / 61.3) with 20, 47.6 / 47.4 (57.7 / 57.5) with 23.
    // The other CTAs share the rest, a warp a domain, when there are enough.
    const uint32_t n3 = !WIDE && M.levels > 3 ? M.num_domains - S.t.level_domain[3] : 0;
    const uint32_t n2 = WIDE ? 0 : whole - n3, nb2 = n2 > kLoopGroup ? (n2 + 2) / 3 : n2;
    const uint32_t skip = !WIDE && n3 + nb2 < blocks / 2 ? n3 + nb2 : 0;
    const uint32_t workers = blocks - skip;
    auto whole_end = [&](uint32_t vb) { return skip && vb >= skip ? 0 : whole; };
    auto first_job = [&](uint32_t vb) {
      return !WIDE && warp < (int)P.gemv_warps && vb >= skip ? warp * workers + (vb - skip) : first2;
    };
    LoopTilesAhead ahead;
    {
      const uint32_t job = first_job(blockIdx.x);
      if (blockIdx.x < whole_end(blockIdx.x)) loop_prefetch(M, M.num_domains - 1 - blockIdx.x, ahead.t[0]);
      else if (job < first2) ahead.first(M, job < n1 ? first1 + job : job - n1);
    }
    if (!loop_barrier(P, S)) break;
    // C
    k = 0;
    for (uint32_t vb = blockIdx.x; vb < blocks; vb += gridDim.x, ++k) {
      double acc = 0.0;
      // `ahead` holds the first tiles of the CTA's first virtual CTA
      const uint32_t end = whole_end(vb), step = !skip ? blocks : (vb < n3 ? whole : nb2);
      for (uint32_t w = vb; w < end; w += step) {
        const uint32_t d = M.num_domains - 1 - w;
        uint32_t l = 0;
        while (l + 1 < M.levels && d >= S.t.level_domain[l + 1]) ++l;
        if (w != blockIdx.x) loop_prefetch(M, d, ahead.t[0]);
        if (l >= 2) loop_coarse(P, d, l, coarse);
        const double* res = l >= 2 ? coarse : (l == 1 ? M.rl64 : P.r);
        const uint32_t base = l >= 2 ? M.level_node_offset[2] : 0u;
        if constexpr (WIDE)
          acc += loop_gemv_cta<double>(P, d, ahead.t[0], res, base, (double)M.weight[l], loop_areas, P.zl64);
        else
          acc += loop_gemv_cta<float>(P, d, ahead.t[0], res, base, (double)M.weight[l], loop_areas, M.zl);
      }
      if constexpr (!WIDE) {
        float4* const area = loop_areas + (size_t)warp * P.area;
        const uint32_t job = first_job(vb);
        const bool fresh = vb == blockIdx.x && vb >= end;  // `ahead` still holds the first job's tiles
        for (uint32_t j = job; j < first2; j += P.gemv_warps * workers) {
          const bool one = j < n1;  // the level-1 domains first
          const uint32_t d = one ? first1 + j : j - n1;
          if (j != job || !fresh) ahead.first(M, d);
          acc += loop_gemv(P, d, ahead, one ? M.rl64 : P.r, 0u, (double)M.weight[one ? 1 : 0], area);
        }
      }
      loop_part(parts, k, acc);
      if constexpr (!SHARED) break;
    }
    loop_parts_end<SHARED>(blocks, parts, P.partials + blocks);
    if (!loop_barrier(P, S)) break;
    // the first z of D while the totals are summed
    double z[3] = {0.0, 0.0, 0.0}, pold[3] = {0.0, 0.0, 0.0};
    const uint32_t d_i = blockIdx.x * kLoopThreads + threadIdx.x;
    if (d_i < M.nv) {
      loop_collect<WIDE>(P, d_i, z);
#pragma unroll
      for (int k = 0; k < 3; ++k) pold[k] = P.p[3ull * d_i + k];
    }
    const double delta = loop_total(P.partials + blocks, blocks), rr = loop_total(P.partials + 2 * blocks, blocks);
    double beta = 0.0;
    int status = kContinue;
    const double it = S.it + 1.0;
    // mas/pcg.py:80-98
    if (!isfinite(delta) || delta < 0.0 || !isfinite(prev) || prev <= 0.0) {
      status = kNonSpd;
    } else {
      beta = restart ? 0.0 : delta / prev;
      const bool done = P.stop_rule == YS_STOP_RESIDUAL ? rr <= st[kTolAbs] : delta <= st[kTolAbs];
      if (done) status = kConverged;
      else if (delta == 0.0) status = kNonSpd;
      else if (it >= st[kMaxItParam]) status = kMaxIter;
    }
    __syncthreads();  // every warp has read S.it
    if (threadIdx.x == 0) {
      S.delta = delta;
      S.prev = prev;
      S.rr = rr;
      S.curv = curv;
      S.alpha = alpha;
      S.beta = beta;
      S.it = it;
      S.status = status;
    }
    if (status != kContinue) break;
    // D
    {
      for (uint32_t i = d_i; i < M.nv; i += gridDim.x * kLoopThreads) {
        if (i != d_i) {
          loop_collect<WIDE>(P, i, z);
#pragma unroll
          for (int k = 0; k < 3; ++k) pold[k] = P.p[3ull * i + k];
        }
        double p[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          p[k] = z[k] + pold[k] * beta;
          P.p[3ull * i + k] = p[k];
        }
        if (sizeof(T) == 4) P.p32[i] = make_float4((float)p[0], (float)p[1], (float)p[2], 0.0f);
      }
    }
    if (!loop_barrier(P, S)) break;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st[kDeltaNew] = S.delta;
    st[kDeltaOld] = S.prev;
    st[kCurv] = S.curv;
    st[kAlpha] = S.alpha;
    st[kBeta] = S.beta;
    st[kRR] = S.rr;
    st[kIter] = S.it;
    st[kStatus] = (double)S.status;
  }
}

// The table of the long rows (and of the levels' domains) from the row plan as
// it stands: one CTA, a contiguous run of rows a thread, so that the segments
// are ordered by row whatever the counts are.  It runs beside the nodes that
// form the first residual, off the solve's critical path.  Where a plan has
// more segments than there is room for, the threshold and the segments double
// until they fit (in the end no row is split).
constexpr int kTableThreads = 1024;

__global__ void __launch_bounds__(kTableThreads) loop_tables_kernel(const __grid_constant__ LoopParams P) {
  __shared__ uint32_t scan[2][kTableThreads / 32];
  const MasDev& M = P.M;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t per = (M.nv + kTableThreads - 1) / kTableThreads;
  const uint32_t r0 = min(M.nv, threadIdx.x * per), r1 = min(M.nv, r0 + per);
  uint32_t threshold = kLongRow, longs, segs, before_longs, before_segs, all_longs, all_segs;
  while (true) {
    longs = segs = 0;
#pragma unroll 4
    for (uint32_t i = r0; i < r1; ++i) {
      uint32_t n = 0;
      for (int s = 0; s < P.nsets; ++s) {
        const uint32_t len = P.sets[s].row_ptr[i + 1] - P.sets[s].row_ptr[i];
        if (len > threshold) n += (len - 1) / (2 * threshold) + 1;
      }
      segs += n;
      longs += n != 0;
    }
    // exclusive sums over the threads
    before_longs = longs;
    before_segs = segs;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t a = __shfl_up_sync(0xffffffffu, before_longs, o), b = __shfl_up_sync(0xffffffffu, before_segs, o);
      if (lane >= o) {
        before_longs += a;
        before_segs += b;
      }
    }
    if (lane == 31) {
      scan[0][warp] = before_longs;
      scan[1][warp] = before_segs;
    }
    __syncthreads();
    before_longs -= longs;
    before_segs -= segs;
    all_longs = all_segs = 0;
    for (int w = 0; w < kTableThreads / 32; ++w) {
      if (w == warp) {
        before_longs += all_longs;
        before_segs += all_segs;
      }
      all_longs += scan[0][w];
      all_segs += scan[1][w];
    }
    if (all_segs <= P.max_segments || threshold >= 1u << 30) break;
    threshold *= 2;
    __syncthreads();  // scan is read
  }
  if (all_segs > P.max_segments) {  // (a row of 2^30 entries: no plan holds one)
    all_longs = all_segs = 0;
    threshold = 0xffffffffu;
  }
  if (threadIdx.x == 0) {
    P.table->threshold = threshold;
    P.table->num_segments = all_segs;
    P.table->num_long = all_longs;
    P.long_first[all_longs] = all_segs;
  }
  if (threadIdx.x <= M.levels) {  // lower bound of the level's first node
    const uint32_t node = M.level_node_offset[threadIdx.x];
    uint32_t lo = 0, hi = M.num_domains;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) / 2;
      if (M.dom_node_ptr[mid] < node) lo = mid + 1;
      else hi = mid;
    }
    P.table->level_domain[threadIdx.x] = lo;
  }
  if (all_longs == 0) return;
  if (longs) {
    for (uint32_t i = r0; i < r1; ++i) {
      uint32_t n = 0;
      for (int s = 0; s < P.nsets; ++s) {
        const uint32_t len = P.sets[s].row_ptr[i + 1] - P.sets[s].row_ptr[i];
        if (len > threshold) n += (len - 1) / (2 * threshold) + 1;
      }
      if (!n) continue;
      P.long_row[before_longs] = i;
      P.long_first[before_longs++] = before_segs;
      before_segs += n;
    }
  }
  __syncthreads();
  for (uint32_t k = warp; k < all_longs; k += kTableThreads / 32) {  // a warp a row
    const uint32_t i = P.long_row[k];
    uint32_t at = P.long_first[k];
    for (int s = 0; s < P.nsets; ++s) {
      const uint32_t e0 = P.sets[s].row_ptr[i], e1 = P.sets[s].row_ptr[i + 1];
      if (e1 - e0 <= threshold) continue;
      const uint32_t n = (e1 - e0 - 1) / (2 * threshold) + 1;
      for (uint32_t j = lane; j < n; j += 32) {
        const uint32_t e = e0 + j * 2 * threshold;
        P.segments[at + j] = make_uint4(i, e, min(e1, e + 2 * threshold), (uint32_t)s);
      }
      at += n;
    }
  }
}

}  // namespace ys
