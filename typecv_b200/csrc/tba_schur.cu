// Structure and values of the explicit reduced camera system (tba_schur.cuh), sm_100a, FP64.
//
//   k_pairs_count   per camera chunk: how many pairs its observations form with each later camera
//   k_pairs_rows    per camera: the camera pairs that occur, into the bit matrix; the row's totals
//   k_pairs_scan    offsets of the rows' camera pairs, observation pairs and blocks of S
//   k_pairs_place   per camera: its camera pairs with their first pairs, each chunk's positions, and
//                   the cameras of its blocks of S
//   k_pairs_blocks  per camera pair: its two blocks of S; the segments that start in it
//   k_pairs_fill    per camera chunk: its pairs, at their positions (within a chunk's share of a camera
//                   pair in the order its threads come: an atomic cursor)
//   k_block_sums    per segment of pairs: sum A_i A_j^T of each camera pair
//   k_block_ends    camera pairs that cross segments: their partial sums in segment order
#include <cuda_runtime.h>

#include "tba_launch.cuh"
#include "tba_schur.cuh"
#include "tba_warp.cuh"

namespace tba {
namespace {

constexpr int kPairThreads = 256;

// A block's problem and its place in that problem's grid: the kernel's argument, or a batch's list.
template <class W>
struct SchurSlot {};
template <>
struct SchurSlot<SchurMany> {
  SchurParams p;
};
__device__ inline const SchurParams& block_problem(const SchurParams& Q, SchurSlot<SchurParams>&, uint32_t& bid) {
  bid = blockIdx.x;
  return Q;
}
__device__ inline const SchurParams& block_problem(const SchurMany& W, SchurSlot<SchurMany>& slot, uint32_t& bid) {
  const uint2 w = W.work[blockIdx.x];
  static_assert(sizeof(SchurParams) % 8 == 0, "copied as 8-byte words");
  const uint64_t* from = reinterpret_cast<const uint64_t*>(W.params + w.x);
  uint64_t* to = reinterpret_cast<uint64_t*>(&slot.p);
  for (uint32_t k = threadIdx.x; k < sizeof(SchurParams) / 8; k += blockDim.x) to[k] = from[k];
  __syncthreads();
  bid = w.y;
  return slot.p;
}

// Calls f(camera of j, j) for every pair (i, j) that the observation at position k of the
// camera-major list contributes to its camera's row: later variable cameras of the same point, and a
// later observation of the same camera (a point seen twice by one camera).
template <typename F>
__device__ inline void row_pairs(const SchurParams& Q, uint32_t k, uint32_t c, F f) {
  const uint32_t i = Q.camera_obs[k], pt = Q.obs_point[i];
  const uint32_t b = Q.point_start[pt], e = Q.point_start[pt + 1];
  for (uint32_t j = b; j < e; j++) {
    const uint32_t d = Q.obs_camera[j];
    if ((d > c && Q.active[d] != 0) || (d == c && j > i)) f(d, i, j);
  }
}

template <class W>
__global__ void __launch_bounds__(kPairThreads) k_pairs_count(W w) {
  after_previous();
  __shared__ SchurSlot<W> slot;
  uint32_t bid;
  const SchurParams& Q = block_problem(w, slot, bid);
  extern __shared__ uint32_t hist[];
  const uint32_t ch = bid, c = Q.chunk_cam[ch];
  if (Q.active[c] == 0) return;
  for (uint32_t d = c + threadIdx.x; d < Q.C; d += blockDim.x) hist[d] = 0;
  __syncthreads();
  const uint32_t end = Q.chunk_beg[ch + 1];
  for (uint32_t k = Q.chunk_beg[ch] + threadIdx.x; k < end; k += blockDim.x)
    row_pairs(Q, k, c, [&](uint32_t d, uint32_t, uint32_t) { atomicAdd(hist + d, 1u); });
  __syncthreads();
  for (uint32_t d = c + threadIdx.x; d < Q.C; d += blockDim.x) Q.counts[size_t(ch) * Q.C + d] = hist[d];
}

// Pairs of row c with camera d, over the row's chunks.
__device__ inline uint32_t row_count(const SchurParams& Q, uint32_t c, uint32_t d) {
  uint32_t n = 0;
  for (uint32_t ch = Q.cam_chunk[c]; ch < Q.cam_chunk[c + 1]; ch++) n += Q.counts[size_t(ch) * Q.C + d];
  return n;
}

template <class W>
__global__ void __launch_bounds__(kPairThreads) k_pairs_rows(W w) {
  after_previous();
  __shared__ SchurSlot<W> slot;
  uint32_t bid;
  const SchurParams& Q = block_problem(w, slot, bid);
  __shared__ uint32_t sum[2];
  const uint32_t c = bid;
  if (threadIdx.x < 2) sum[threadIdx.x] = 0;
  if (threadIdx.x == 0) atomicOr(Q.bits + size_t(c) * Q.bwords + c / 32, 1u << (c % 32));
  __syncthreads();
  if (Q.active[c] != 0) {
    uint32_t blocks = 0, pairs = 0;
    for (uint32_t d = c + threadIdx.x; d < Q.C; d += blockDim.x) {
      const uint32_t n = row_count(Q, c, d);
      if (n == 0) continue;
      blocks++;
      pairs += n;
      if (d != c) {
        atomicOr(Q.bits + size_t(c) * Q.bwords + d / 32, 1u << (d % 32));
        atomicOr(Q.bits + size_t(d) * Q.bwords + c / 32, 1u << (c % 32));
      }
    }
    atomicAdd(sum, blocks);
    atomicAdd(sum + 1, pairs);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    Q.row_blk[c] = sum[0];
    Q.row_pair[c] = sum[1];
  }
}

// Exclusive scan of N values over the block's threads; `total` receives the sums.
template <int N>
__device__ inline void block_scan(uint32_t (&v)[N], uint32_t (&total)[N], uint32_t (*warp_sum)[N]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t own[N];
#pragma unroll
  for (int n = 0; n < N; n++) own[n] = v[n];
  for (int d = 1; d < 32; d <<= 1)
#pragma unroll
    for (int n = 0; n < N; n++) {
      const uint32_t t = __shfl_up_sync(kFull, v[n], d);
      if (lane >= d) v[n] += t;
    }
  __syncthreads();
  if (lane == 31)
#pragma unroll
    for (int n = 0; n < N; n++) warp_sum[warp][n] = v[n];
  __syncthreads();
#pragma unroll
  for (int n = 0; n < N; n++) {
    uint32_t before = 0, all = 0;
    for (int w = 0; w < nw; w++) {
      const uint32_t s = warp_sum[w][n];
      if (w < warp) before += s;
      all += s;
    }
    v[n] += before - own[n];
    total[n] = all;
  }
  __syncthreads();
}

template <class W>
__global__ void __launch_bounds__(1024) k_pairs_scan(W w) {
  after_previous();
  __shared__ SchurSlot<W> slot;
  uint32_t bid;
  const SchurParams& Q = block_problem(w, slot, bid);
  __shared__ uint32_t warp_sum[32][3];
  uint32_t base[3] = {0, 0, 0};
  for (uint32_t c0 = 0; c0 < Q.C; c0 += blockDim.x) {
    const uint32_t c = c0 + threadIdx.x;
    uint32_t v[3] = {0, 0, 0}, total[3];
    if (c < Q.C) {
      v[0] = Q.row_blk[c];
      v[1] = Q.row_pair[c];
      for (uint32_t w = 0; w < Q.bwords; w++) v[2] += __popc(Q.bits[size_t(c) * Q.bwords + w]);
    }
    block_scan(v, total, warp_sum);
    if (c < Q.C) {
      Q.row_blk[c] = base[0] + v[0];
      Q.row_pair[c] = base[1] + v[1];
      Q.row_ptr[c] = base[2] + v[2];
    }
    for (int n = 0; n < 3; n++) base[n] += total[n];
  }
  if (threadIdx.x == 0) {
    Q.row_blk[Q.C] = Q.totals[0] = base[0];
    Q.row_pair[Q.C] = Q.totals[1] = base[1];
    Q.row_ptr[Q.C] = Q.totals[2] = base[2];
    Q.blk_begin[base[0]] = base[1];
  }
}

template <class W>
__global__ void __launch_bounds__(kPairThreads) k_pairs_place(W w) {
  after_previous();
  __shared__ SchurSlot<W> slot;
  uint32_t bid;
  const SchurParams& Q = block_problem(w, slot, bid);
  __shared__ uint32_t warp_sum[kPairThreads / 32][2];
  const uint32_t c = bid;
  // The cameras of the row's blocks, in order.
  uint32_t at = Q.row_ptr[c];
  for (uint32_t w0 = 0; w0 < Q.bwords; w0 += blockDim.x) {
    const uint32_t w = w0 + threadIdx.x;
    uint32_t word = w < Q.bwords ? Q.bits[size_t(c) * Q.bwords + w] : 0u;
    uint32_t v[2] = {uint32_t(__popc(word)), 0}, total[2];
    block_scan(v, total, warp_sum);
    uint32_t to = at + v[0];
    for (; word; word &= word - 1) Q.col[to++] = 32 * w + uint32_t(__ffs(word) - 1);
    at += total[0];
  }
  if (Q.active[c] == 0) return;
  uint32_t blk = Q.row_blk[c], pair = Q.row_pair[c];
  for (uint32_t d0 = c; d0 < Q.C; d0 += blockDim.x) {
    const uint32_t d = d0 + threadIdx.x, n = d < Q.C ? row_count(Q, c, d) : 0u;
    uint32_t v[2] = {n != 0 ? 1u : 0u, n}, total[2];
    block_scan(v, total, warp_sum);
    if (n) {
      const uint32_t b = blk + v[0];
      uint32_t first = pair + v[1];
      Q.blk_begin[b] = first;
      Q.blk_rc[b] = make_uint2(c, d);
      for (uint32_t ch = Q.cam_chunk[c]; ch < Q.cam_chunk[c + 1]; ch++) {
        uint32_t* q = Q.counts + size_t(ch) * Q.C + d;
        const uint32_t k = *q;
        *q = first;
        first += k;
      }
    }
    blk += total[0];
    pair += total[1];
  }
}

// Position of camera d among the blocks of row c.
__device__ inline uint32_t block_of(const SchurParams& Q, uint32_t c, uint32_t d) {
  const uint32_t* row = Q.bits + size_t(c) * Q.bwords;
  uint32_t n = Q.row_ptr[c];
  for (uint32_t w = 0; w < d / 32; w++) n += __popc(row[w]);
  return n + __popc(row[d / 32] & ((1u << (d % 32)) - 1u));
}

template <class W>
__global__ void __launch_bounds__(kPairThreads) k_pairs_blocks(W w) {
  after_previous();
  __shared__ SchurSlot<W> slot;
  uint32_t bid;
  const SchurParams& Q = block_problem(w, slot, bid);
  const uint32_t b = bid * blockDim.x + threadIdx.x;
  if (b >= Q.totals[0]) return;
  const uint2 rc = Q.blk_rc[b];
  Q.blk_dst[b] = make_uint2(block_of(Q, rc.x, rc.y), block_of(Q, rc.y, rc.x));
  const uint32_t begin = Q.blk_begin[b], end = Q.blk_begin[b + 1];
  for (uint32_t s = (begin + Q.seg - 1) / Q.seg; s * Q.seg < end; s++) Q.seg_block[s] = b;
}

template <class W>
__global__ void __launch_bounds__(kPairThreads) k_pairs_fill(W w) {
  after_previous();
  __shared__ SchurSlot<W> slot;
  uint32_t bid;
  const SchurParams& Q = block_problem(w, slot, bid);
  extern __shared__ uint32_t cursor[];
  const uint32_t ch = bid, c = Q.chunk_cam[ch];
  if (Q.active[c] == 0) return;
  for (uint32_t d = c + threadIdx.x; d < Q.C; d += blockDim.x) cursor[d] = Q.counts[size_t(ch) * Q.C + d];
  __syncthreads();
  const uint32_t end = Q.chunk_beg[ch + 1];
  for (uint32_t k = Q.chunk_beg[ch] + threadIdx.x; k < end; k += blockDim.x)
    row_pairs(Q, k, c, [&](uint32_t d, uint32_t i, uint32_t j) { Q.pairs[atomicAdd(cursor + d, 1u)] = make_uint2(i, j); });
}

// One m8n8k4 FP64 matrix instruction: d += a b^T of the lane's fragments (a: row lane / 4, column
// lane % 4; b the same; d: row lane / 4, columns 2 (lane % 4) and the next).
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Entry (r, k) of camera pair b of S: -v in the block of its row and, transposed, of its column.  A
// pair of observations of one camera adds both orders to the diagonal block.
__device__ inline void store_entry(const SchurParams& Q, uint32_t b, uint32_t r, uint32_t k, double v) {
  const uint2 at = Q.blk_dst[b];
  double* own = Q.S + 36 * size_t(at.x) + 6 * k + r;
  double* other = Q.S + 36 * size_t(at.y) + 6 * r + k;
  if (at.x == at.y) {
    atomicAdd(own, -v);
    atomicAdd(other, -v);
    return;
  }
  *own = -v;
  *other = -v;
}

// One segment of pairs per warp.  The columns of the pairs' records follow one another along the
// matrix instruction's inner dimension (four pairs are three instructions); a lane loads its own
// element of each record from global memory, so a record is read as whole 48-byte columns.  The
// segment's pairs come 32 at a time, one a lane, so that a record's loads wait for one load only.  Bound by
// the L1: a record of 144 bytes is two lines, and a load's lanes touch four (1.18 ms for 30M pairs, half of
// the L1's wavefronts on average and three quarters on the busiest SM; DRAM at a fifth).
template <class W>
__global__ void __launch_bounds__(256) k_block_sums(W w) {
  after_previous();
  __shared__ SchurSlot<W> slot;
  uint32_t bid;
  const SchurParams& Q = block_problem(w, slot, bid);
  if (Q.go && *Q.go == 0) return;
  const uint32_t s = bid * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const uint32_t npairs = Q.totals[1];
  const uint32_t lo = s * Q.seg;
  if (lo >= npairs) return;
  const uint32_t hi = min(npairs, lo + Q.seg);
  const int lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
  int off[3];
  uint32_t word[3];
#pragma unroll
  for (int t = 0; t < 3; t++) {
    off[t] = (4 * t + q) / 3;
    word[t] = uint32_t(4 * t + q) % 3 * 6 + r;
  }
  uint32_t b = Q.seg_block[s], begin = Q.blk_begin[b], stop = Q.blk_begin[b + 1];
  const double* const A = Q.A;
  const uint2* const pairs = Q.pairs;
  double d0 = 0, d1 = 0;
  for (uint32_t base = lo; base < hi; base += 32) {
    const uint32_t n = min(32u, hi - base);
    const uint2 mine = uint32_t(lane) < n ? pairs[base + lane] : make_uint2(0, 0);
    for (uint32_t p = base; p < base + n;) {
      const uint32_t e = min(stop, base + n);
#pragma unroll 4
      for (uint32_t g = p; g < e; g += 4) {
        double a[3], c[3];
#pragma unroll
        for (int t = 0; t < 3; t++) {
          const uint32_t k = g + off[t];
          const uint32_t i = __shfl_sync(kFull, mine.x, k - base), j = __shfl_sync(kFull, mine.y, k - base);
          a[t] = c[t] = 0;
          if (r < 6 && k < e) {
            a[t] = A[18 * size_t(i) + word[t]];
            c[t] = A[18 * size_t(j) + word[t]];
          }
        }
#pragma unroll
        for (int t = 0; t < 3; t++) dmma(d0, d1, a[t], c[t]);
      }
      p = e;
      if (e != stop && e != hi) continue;  // the camera pair goes on in the next 32
      if (r < 6 && q < 3) {
        if (begin >= lo && stop <= hi) {
          store_entry(Q, b, r, 2 * q, d0);
          store_entry(Q, b, r, 2 * q + 1, d1);
        } else {  // the camera pair began before this segment (slot 0) or goes on after it (slot 1)
          double* part = Q.part + 36 * (2 * size_t(s) + (begin < lo ? 0 : 1)) + 6 * r + 2 * q;
          *reinterpret_cast<double2*>(part) = make_double2(d0, d1);
        }
      }
      d0 = d1 = 0;
      if (e < hi) {
        b++;
        begin = stop;
        stop = Q.blk_begin[b + 1];
      }
    }
  }
}

// A warp per segment boundary: the camera pair that crosses it, taken at the first of the boundaries it
// crosses.  (A warp per possible camera pair, nearly all with nothing to do: 88 us at 1,500 cameras; 20.)
template <class W>
__global__ void __launch_bounds__(256) k_block_ends(W w) {
  after_previous();
  __shared__ SchurSlot<W> slot;
  uint32_t bid;
  const SchurParams& Q = block_problem(w, slot, bid);
  if (Q.go && *Q.go == 0) return;
  const uint32_t s = bid * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const uint64_t lo = uint64_t(s) * Q.seg;
  if (s == 0 || lo >= Q.totals[1]) return;
  const uint32_t b = Q.seg_block[s], begin = Q.blk_begin[b], end = Q.blk_begin[b + 1];
  const uint32_t s0 = begin / Q.seg, s1 = (end - 1) / Q.seg;
  if (begin >= lo || s0 != s - 1) return;
  // An entry a lane, and the last four with the first lanes' (together: their loads wait once).
  const uint32_t e = threadIdx.x & 31;
  const double* part = Q.part + 36 * (2 * size_t(s0) + 1) + e;
  const bool two = e < 4;
  double v = part[0], u = two ? part[32] : 0.0;
  part -= 36;
#pragma unroll 4
  for (uint32_t k = s0 + 1; k <= s1; k++) {
    part += 72;
    v += part[0];
    if (two) u += part[32];
  }
  store_entry(Q, b, e / 6, e % 6, v);
  if (two) store_entry(Q, b, 5, e + 2, u);
}

}  // namespace

uint32_t schur_launch_structure(const SchurParams& q, cudaStream_t s) {
  const size_t smem = size_t(q.C) * sizeof(uint32_t);
  cudaMemsetAsync(q.bits, 0, size_t(q.C) * q.bwords * sizeof(uint32_t), s);
  launch_dependent(k_pairs_count<SchurParams>, q.nchunks, kPairThreads, smem, s, q);
  launch_dependent(k_pairs_rows<SchurParams>, q.C, kPairThreads, 0, s, q);
  launch_dependent(k_pairs_scan<SchurParams>, 1, 1024, 0, s, q);
  launch_dependent(k_pairs_place<SchurParams>, q.C, kPairThreads, 0, s, q);
  if (q.max_blocks) launch_dependent(k_pairs_blocks<SchurParams>, (q.max_blocks + kPairThreads - 1) / kPairThreads, kPairThreads, 0, s, q);
  launch_dependent(k_pairs_fill<SchurParams>, q.nchunks, kPairThreads, smem, s, q);
  return q.max_blocks ? 6 : 5;
}

uint32_t schur_launch_values(const SchurParams& q, cudaStream_t s) {
  if (!q.max_pairs) return 0;
  const uint32_t segs = (q.max_pairs + q.seg - 1) / q.seg;
  launch_dependent(k_block_sums<SchurParams>, (segs + 7) / 8, 256, 0, s, q);
  launch_dependent(k_block_ends<SchurParams>, (segs + 7) / 8, 256, 0, s, q);
  return 2;
}

uint32_t schur_launch_many_structure(const SchurLists& b, cudaStream_t s) {
  const size_t smem = size_t(b.max_cameras) * sizeof(uint32_t);
  k_pairs_count<SchurMany><<<b.chunk.blocks, kPairThreads, smem, s>>>(b.chunk.of(b));
  k_pairs_rows<SchurMany><<<b.camera.blocks, kPairThreads, 0, s>>>(b.camera.of(b));
  k_pairs_scan<SchurMany><<<b.one.blocks, 1024, 0, s>>>(b.one.of(b));
  k_pairs_place<SchurMany><<<b.camera.blocks, kPairThreads, 0, s>>>(b.camera.of(b));
  k_pairs_blocks<SchurMany><<<b.pairs.blocks, kPairThreads, 0, s>>>(b.pairs.of(b));
  k_pairs_fill<SchurMany><<<b.chunk.blocks, kPairThreads, smem, s>>>(b.chunk.of(b));
  return 6;
}

uint32_t schur_launch_many_values(const SchurLists& b, cudaStream_t s) {
  k_block_sums<SchurMany><<<b.sums.blocks, 256, 0, s>>>(b.sums.of(b));
  k_block_ends<SchurMany><<<b.sums.blocks, 256, 0, s>>>(b.sums.of(b));
  return 2;
}

}  // namespace tba
