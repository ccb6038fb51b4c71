// The explicit reduced camera system: the point-eliminated Schur complement
//   S_cd = [c = d] U_c - sum_{i in c, j in d, same point p} W_i V_p^-1 W_j^T
// formed once per linear solve as a block-sparse symmetric matrix over the cameras (plus the shared
// focal column), so that a PCG step multiplies by S instead of passing over every observation.
//
// With V_p^-1 = N_p N_p^T the block of a pair of observations of one point is A_i A_j^T with the
// 6x3 record A_i = W_i N_p, so S is formed from the records alone.
//
//   structure (once per call): the pairs (i, j) of observations of one point in two variable
//     cameras, c(i) < c(j), grouped by camera pair; the camera pairs that occur (a bit matrix), and
//     the rows of S as runs of 6x6 blocks in camera order
//   values (per solve): every camera pair's sum of A_i A_j^T on the FP64 matrix instruction, in
//     equal runs of pairs per warp whose unfinished ends are added afterwards in the runs' order.  The
//     pairs of a camera pair lie in the order in which k_pairs_fill's atomic cursor met them, which
//     changes from call to call: S repeats to rounding, not bit for bit
//   PCG: one persistent launch per run (tba_pcg.cu)
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace tba {

constexpr uint32_t kPairSegMin = 32, kPairSegMax = 512;  // pairs per warp of the block sums

struct SchurParams {
  uint32_t C, M, nchunks;
  uint32_t bwords;     // words of a row of the bit matrix
  uint32_t seg;        // pairs per warp of the block sums
  uint32_t max_pairs;  // the host's bound on the pairs (fixed cameras included)
  uint32_t max_blocks; // the host's bound on the camera pairs
  // The problem's index sections and camera chunks.
  const uint32_t* obs_camera;
  const uint32_t* obs_point;
  const uint32_t* point_start;
  const uint32_t* camera_obs;
  const uint32_t* active;
  const uint32_t* chunk_cam;
  const uint32_t* chunk_beg;
  const uint32_t* cam_chunk;
  // Structure.
  uint32_t* counts;     // nchunks x C: pairs of the chunk's observations with each camera, then their positions
  uint32_t* bits;       // C x bwords: the camera pairs of S (symmetric, diagonal included)
  uint32_t* row_blk;    // C + 1: first camera pair of each row of the upper triangle
  uint32_t* row_pair;   // C + 1: first observation pair
  uint32_t* row_ptr;    // C + 1: first block of each row of S
  uint32_t* col;        // camera of each block of S, ascending in a row
  uint2* pairs;         // observations (i, j)
  uint32_t* blk_begin;  // max_blocks + 1: first pair of each camera pair
  uint2* blk_rc;        // its cameras
  uint2* blk_dst;       // its blocks in the two rows of S
  uint32_t* seg_block;  // camera pair of each segment's first pair
  uint32_t* totals;     // camera pairs, observation pairs, blocks of S
  // Values (nothing is done while *go is zero).
  const double* go;
  double* A;     // 18 per observation: W_i N_p by columns ([k * 6 + row])
  double* part;  // 2 x 36 per segment: the sums of camera pairs that cross segments
  double* S;     // 36 per block, by columns (entry (row a, column b) at 6 b + a)
};

// The same over a batch: every problem's parameters in device memory, and lists of (problem, block).
struct SchurMany {
  const SchurParams* params;
  const uint2* work;
};
struct SchurLists {
  const SchurParams* params;
  uint32_t max_cameras;
  struct List {
    const uint2* work;
    uint32_t blocks;
    SchurMany of(const SchurLists& b) const { return SchurMany{b.params, work}; }
  };
  // A block per: problem; camera chunk; camera; 256 camera pairs; eight segments.
  List one, chunk, camera, pairs, sums;
};
uint32_t schur_launch_many_structure(const SchurLists& b, cudaStream_t s);  // (bits zeroed by the caller)
uint32_t schur_launch_many_values(const SchurLists& b, cudaStream_t s);

// Structure of S (indices already checked), on stream s; returns the kernels launched.
uint32_t schur_launch_structure(const SchurParams& q, cudaStream_t s);
// The off-diagonal blocks of S from the records; returns the kernels launched.
uint32_t schur_launch_values(const SchurParams& q, cudaStream_t s);

}  // namespace tba
