// Device-resident restarted GMRES (left preconditioned), restating
// jax.scipy.sparse.linalg.gmres as called at steppers.py:466 / :476.
#pragma once

#include "sisl_core.cuh"

namespace sisl {

constexpr int GM_MAXR = 128;     // largest supported restart (Krylov) dimension
constexpr int GM_MAXBLOCKS = 1184;  // 8 * 148 SMs: reduction partials per kernel
constexpr int GM_S = 6;          // largest number of basis vectors formed per orthogonalisation
constexpr int GM_BLOCKS = 2 * 148;  // grid of the block kernels: two resident blocks per SM
constexpr int GM_GROUP = 16;     // blocks per first-level group of the block dots' reduction

// Scalars and small dense matrices of one solve, all float64, in workspace.
//
// In the block form the Krylov basis Q is kept as stored vectors V and a block-diagonal upper
// triangular factor: Q_l = sum_q B[l][q] V_{bstart[l] + q}.  The vectors of
// one block are orthogonalised together (sisl_gmres.cu).
struct GState {
  double h[GM_MAXR + 2];            // projections of the new vector (scaled; one column per block)
  double s[GM_MAXR + 2];            // scale of V_j as operator input (one column per block: its inverse norm)
  double B[GM_MAXR + 2][GM_S];      // Q_l in the stored vectors of its block
  int bstart[GM_MAXR + 2];          // first stored vector of Q_l's block
  double H[GM_MAXR][GM_MAXR + 1];   // Hessenberg rows (batched) or rotated R rows (incremental)
  double hraw[GM_MAXR][GM_MAXR + 1];  // Hessenberg columns before rotation
  double givens[GM_MAXR][2];
  double beta[GM_MAXR + 1];
  double coef[GM_MAXR + 2];         // coefficients of the end-of-cycle update in the stored vectors
  // the block being orthogonalised (first new vector m = j0 + 1, bs columns kept)
  double r1[GM_MAXR + 1][GM_S];     // Z_i in Q_0 .. Q_j0
  double r2[GM_S][GM_S];            // Z_i in the block's own (not yet corrected) vectors
  double u[GM_S][GM_S];             // inverse of r2
  double cv[GM_MAXR + 1][GM_S];     // new vector i = sum_k u[k][i] Z_k - sum_l cv[l][i] V_l
  double clast[GM_S];               // the last stored vector in its block's Q
  int cstart, clen, bs;
  double hn0;                       // ||M A v_j|| before orthogonalisation (one column per block)
  double bnorm, mbnorm, rnorm, atol, ptol, tol, atol_in, eps;
  double err;                       // incremental residual estimate
  int active;                       // 1 while the current cycle continues
  int kdone;                        // Arnoldi steps taken in the current cycle
  int restart;
  int method;                       // 0 batched, 1 incremental
  int columns;                      // columns per block at most; 1: the classical form
  int breakdown;
  int narrow;                       // a block of this cycle lost columns: the cycle is done over, one column at a time
  unsigned int counter;             // last-block-done ticket
  unsigned int group_counter[GM_BLOCKS / GM_GROUP + 1];
  int cycles, steps;                // restart cycles and Arnoldi steps taken (graph mode)
};

// Columns of each block of a cycle of R steps, at most S (<= GM_S) each:
// equal shares for the batched solve; the incremental one starts with short
// blocks, since a cycle that leaves early has applied the operator for its
// whole last block (a ramp of 2, 4 costs under 3 % more vector traffic at
// R = 30 than equal shares of 6).  Returns the number of blocks.
inline int gm_block_plan(int R, int S, int method, int* cols) {
  int nb = 0, left = R;
  if (method != 0)
    for (int c = 2; c < S && left > 0; c += 2) {
      cols[nb] = c < left ? c : left;
      left -= cols[nb++];
    }
  int parts = (left + S - 1) / S;
  for (; parts > 0; --parts) {
    cols[nb] = (left + parts - 1) / parts;
    left -= cols[nb++];
  }
  return nb;
}
// row tiles (8 rows each) the block dots is instantiated for
inline int gm_row_tiles(int rows) {
  const int inst[] = {1, 2, 3, 4, 5, 6, 8, 10, 13, 17};
  for (int t : inst)
    if (8 * t >= rows) return t;
  return 17;
}
// reduction scratch of one solve, doubles
inline size_t gm_partial_doubles(int R) {
  const size_t dots = (size_t)(GM_BLOCKS + GM_BLOCKS / GM_GROUP + 1) * gm_row_tiles(R + 1) * 64;
  const size_t rest = (size_t)GM_MAXBLOCKS * (GM_MAXR + 2);
  return dots > rest ? dots : rest;
}

// Per-solve statistics written on the device in graph mode; the same layout
// as SislSolveInfo.
struct GDevInfo {
  int32_t cycles, arnoldi_steps, converged, pad;
  double residual_norm, atol, b_norm;
};

// Host-visible summary copied back once per restart cycle.
struct GHostView {
  double rnorm, atol, bnorm;
  int kdone;
  int narrow;
};

}  // namespace sisl
