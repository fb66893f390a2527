// MAS preconditioner hooks used by the PCG graph builder.
#pragma once

#include "ys_pcg.cuh"

namespace ys {

// Launches of the one-kernel loop (mas_pcg_loop) of one solver.  Its sums are
// split among `blocks` virtual CTAs; body b of the solve's switch nodes runs
// them on grid[b] CTAs, and body_of[k - 1] is the body while k solves of the
// process (kLoopShares or more for the last) share the chip.
constexpr int kLoopShares = 4;
struct MasLoopPlan {
  bool used = false, wide = false;
  const void* kernel = nullptr;         // a CTA a virtual one
  const void* shared_kernel = nullptr;  // fewer CTAs
  uint32_t blocks = 0, gemv_warps = 0;
  size_t smem = 0;
  int bodies = 0;
  unsigned grid[kLoopShares] = {};
  int body_of[kLoopShares] = {};
};

struct MasPcgHooks {
  void* params = nullptr;  // owned by the MAS handle
  bool fused_direction = false;  // the loop body's last MAS node also updates p
  MasLoopPlan loop;              // mas_plan_loop's, before any node is added
  double* loop_workspace = nullptr;  // mas_loop_workspace_doubles(num_vars) of the caller's workspace
};

// Nodes computing r = g - H x (or r = g), z = M^-1 r, p = z and the initial
// reductions / stop threshold; sets the loop condition.  `*last` receives the
// final node.
cudaError_t mas_add_init_nodes(void* mas, cudaGraph_t g, const cudaGraphNode_t* deps, size_t ndeps,
                               cudaGraphNode_t* last, uint32_t nv, const double* rhs, double* x, double* r, double* p,
                               float4* p32, double* q, double* z, double* st, double* partials, unsigned* tickets, const SpmvSet* sets,
                               int nsets, int fp32, int stop_rule, int zero_guess, double tolerance, uint32_t max_it,
                               cudaGraphConditionalHandle cond, MasPcgHooks* hooks);

// Nodes of the loop body after spmv_dot: x/r update, z = M^-1 r, r^T z,
// beta and the stop test.
cudaError_t mas_add_update_nodes(void* mas, cudaGraph_t body, const cudaGraphNode_t* deps, size_t ndeps,
                                 cudaGraphNode_t* last, MasPcgHooks* hooks);

// Decides whether the system is small enough for the whole loop as one
// cooperative kernel (loop->used), and its grids.
cudaError_t mas_plan_loop(void* mas, int fp32, MasLoopPlan* loop);

// That kernel as the only node of each of `count` bodies, on the grids from
// loop.grid[first] on.  *tables is the node of `g` that reads the row plan for
// it: the loop has to come after it.
cudaError_t mas_add_loop_nodes(void* mas, cudaGraph_t g, const cudaGraph_t* bodies, int first, int count,
                               cudaGraphNode_t* tables, MasPcgHooks* hooks);

// Doubles of the solve's workspace that the one-kernel loop takes (0 beyond its sizes).
uint64_t mas_loop_workspace_doubles(uint32_t num_vars);

}  // namespace ys
