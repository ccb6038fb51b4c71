// The PCG on an explicit reduced camera system (tba_schur.cuh) as one persistent launch.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace tba {

constexpr uint32_t kPcgWaitPolls = 1u << 21;  // polls of one wait before it gives up, at most (about a second)

// A double and the step it belongs to, written and read as one 16-byte word: a reader that finds the
// step it waits for has the value, with no fence on either side.
struct alignas(16) Flagged {
  double value;
  uint64_t step;
};

// The system, its vectors and the words of the solver's state that the PCG reads and writes.
struct PcgSystem {
  uint32_t C, shared;  // cameras; a focal unknown after the 6C camera unknowns
  const double* S;     // 6x6 blocks by columns: entry (row a, column b) of block k at 36 k + 6 b + a
  const uint32_t* row_ptr;  // C + 1 first blocks of the rows
  const uint32_t* col;      // camera of each block
  // Per block of the launch (pcg_launch_plan): its first camera, its distinct columns' cameras and, per
  // block of S, the place of its camera among them.
  uint32_t* share;     // grid + 1
  uint32_t* uni;       // grid x C
  uint32_t* uni_n;     // grid
  uint32_t* local;     // per block of S
  const double* Minv;  // 36C block-Jacobi preconditioner
  const double* scf;   // 6C focal column (with the focal unknown)
  double *x, *r, *z, *p;  // 6C (+ 1); x and r are updated, z and p hold the start (p = z or a restart's)
  double* pbuf;           // grid x 2 x 6C: a block's direction and its columns' z when they do not fit shared memory
  double* state;
  int active, failed, converged, rho, r0, r2, inner_r0, steps, all_steps, wait;  // words; -1: not kept
  int focal_diag, focal_inv;
  // With `rhs` (6C) the run starts itself: r = rhs, x = 0, z = M^-1 r, the focal unknown from the task
  // blocks' partial sums, and the start's words (k_pcg_init does the same for steps launched one by one).
  const double* rhs;
  const double* scal_part;  // 4 per task block: H_ff, b_f, and the points' shares of them
  uint32_t scal_blocks;
  uint32_t max_blocks;      // 6x6 blocks of S at most
  int solving, block_failed, lambda, focal_full, focal_rhs, clear_from, clear_to;
  uint32_t polls;           // of one wait for other blocks (at most kPcgWaitPolls)
  double tol, tol_inner, alpha_limit;
  Flagged* zx;         // 6C: z between blocks
  Flagged* slots;      // 4 per block: its partial sums of the step's two reductions
};

cudaError_t pcg_configure();
// Blocks of a run on a system of at most `blocks` 6x6 blocks.
uint32_t pcg_grid(uint64_t blocks, uint32_t C, int sms);
// The blocks' shares and columns, once per structure.
uint32_t pcg_launch_plan(const PcgSystem& a, uint32_t grid, cudaStream_t s);
// Up to `limit` PCG steps from the vectors and state as k_pcg_init (or a restart) left them.
cudaError_t launch_pcg(const PcgSystem& a, uint32_t limit, uint32_t grid, cudaStream_t s);

// The systems of a batch, one block each (list: problem of each block).
struct PcgMany {
  const PcgSystem* systems;
  const uint2* work;
};
uint32_t pcg_launch_many_plan(const PcgMany& b, uint32_t count, uint32_t max_cameras, cudaStream_t s);
cudaError_t launch_many_pcg(const PcgMany& b, uint32_t count, bool shared, uint32_t limit, cudaStream_t s);

}  // namespace tba
