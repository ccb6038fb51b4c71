// The persistent PCG (tba_pcg.cuh), sm_100a, FP64.
//
// Each block owns a run of cameras (about the same number of 6x6 blocks of S each) and keeps in shared
// memory, as far as they fit, its rows of S, the direction p of the cameras its rows touch, and its
// shares of x, r and S p.  A step is
//   p = z + beta p of the block's columns, S p of its rows, p . S p          -> sum over the grid, alpha
//   x += alpha p, r -= alpha S p, z = M^-1 r of its own cameras, r.r, z.r    -> sum over the grid, beta
// and only z and four partial sums a block cross between blocks, as values that carry their step's
// number (Flagged): no barrier, no fence, and the L1 keeps what the step only reads.  Every block adds
// the partial sums in the same order, so all take the same decisions.  A block can publish a step's z
// only once every block has published the sums that follow its use of the last z, and a reduction's
// sums only after the other reduction (the start counts as a second one), so one buffer of each does.
// What bounds a step is the two exchanges through the L2 (1.6 us each between 22 blocks, 2.0 to 2.7 between
// 148, with the wait for the slowest block), and the block's own chain of reductions, divisions and barriers
// (2.6 us at 7 cameras in one block).
#include <cuda_runtime.h>

#include <algorithm>

#include "tba_launch.cuh"
#include "tba_pcg.cuh"
#include "tba_warp.cuh"

namespace tba {
namespace {

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr uint32_t kSmemBytes = 208 * 1024;

__device__ __forceinline__ void publish(Flagged* p, double v, uint64_t step) {
  asm volatile(
      "{\n .reg .b128 w;\n mov.b128 w, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], w;\n}" ::"l"(p),
      "l"(__double_as_longlong(v)), "l"(step)
      : "memory");
}

__device__ __forceinline__ Flagged peek(const Flagged* p) {
  uint64_t v, s;
  asm volatile("{\n .reg .b128 w;\n ld.relaxed.gpu.global.b128 w, [%2];\n mov.b128 {%0, %1}, w;\n}"
               : "=l"(v), "=l"(s)
               : "l"(p)
               : "memory");
  return Flagged{__longlong_as_double(v), s};
}

// The values of `step` at N places, looked for together (a place beyond `n` is left out); false when
// they did not come within `polls` polls.
template <int N>
__device__ __forceinline__ bool await(const Flagged* const (&p)[N], int n, uint64_t step, uint32_t polls, double (&v)[N]) {
  for (uint32_t k = 0; k < polls; k++) {
    Flagged f[N];
#pragma unroll
    for (int j = 0; j < N; j++)
      if (j < n) f[j] = peek(p[j]);
    bool all = true;
#pragma unroll
    for (int j = 0; j < N; j++)
      if (j < n) {
        all = all && f[j].step == step;
        v[j] = f[j].value;
      }
    if (all) return true;
  }
  return false;
}

// A block's system and its place in that system's grid: the kernel's argument, or a batch's list (one
// block a system).
template <class W>
struct PcgSlot {};
template <>
struct PcgSlot<PcgMany> {
  PcgSystem a;
};
__device__ inline const PcgSystem& block_system(const PcgSystem& A, PcgSlot<PcgSystem>&, uint32_t& bid, uint32_t& grid) {
  bid = blockIdx.x;
  grid = gridDim.x;
  return A;
}
__device__ inline const PcgSystem& block_system(const PcgMany& W, PcgSlot<PcgMany>& slot, uint32_t& bid, uint32_t& grid) {
  static_assert(sizeof(PcgSystem) % 8 == 0, "copied as 8-byte words");
  const uint64_t* from = reinterpret_cast<const uint64_t*>(W.systems + W.work[blockIdx.x].x);
  uint64_t* to = reinterpret_cast<uint64_t*>(&slot.a);
  for (uint32_t k = threadIdx.x; k < sizeof(PcgSystem) / 8; k += blockDim.x) to[k] = from[k];
  __syncthreads();
  bid = 0;
  grid = 1;
  return slot.a;
}

struct Shared {
  double red[2][kWarps][2];
  double part[kWarps][6];
  double sum[2];
  int gave_up;
};

constexpr int kSlotsEach = 5;  // partial sums of 32 x 5 blocks in one round of a warp (148 SMs)

// Adds v, which only the first `warps` warps have, over the grid; every thread returns with the sums
// (false: a wait gave up).  `which` is the step's first or second reduction.  While the first warp
// waits for the other blocks' sums, the others run `meanwhile`.
template <class F>
__device__ inline bool grid_sum(const PcgSystem& A, Shared& sh, double (&v)[2], uint64_t step, int which, int warps,
                                uint32_t bid, uint32_t grid, F meanwhile) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < warps) {
    warp_allsum(v);
    if (lane == 0) {
      sh.red[which][warp][0] = v[0];
      sh.red[which][warp][1] = v[1];
    }
  }
  __syncthreads();
  if (grid == 1) {
    v[0] = v[1] = 0;
    for (int w = 0; w < warps; w++) {
      v[0] += sh.red[which][w][0];
      v[1] += sh.red[which][w][1];
    }
    return true;
  }
  if (warp == 0) {
    double t[2] = {lane < warps ? sh.red[which][lane][0] : 0.0, lane < warps ? sh.red[which][lane][1] : 0.0};
    if (warps > 1) warp_allsum(t);
    Flagged* slots = A.slots + 2 * size_t(which);
    t[1] = __shfl_sync(kFull, t[1], 0);  // lane 1 publishes the second sum
    if (lane < 2) publish(slots + 4 * size_t(bid) + lane, lane == 0 ? t[0] : t[1], step);
    bool ok = *(volatile int*)&sh.gave_up == 0;
    double s[2] = {0, 0};
    for (uint32_t base = 0; base < grid && ok; base += 32 * kSlotsEach) {
      const Flagged* at[2 * kSlotsEach];
      double got[2 * kSlotsEach];
      int n = 0;
#pragma unroll
      for (int j = 0; j < kSlotsEach; j++) {
        const uint32_t b = base + 32 * j + lane;
        at[2 * j] = slots + 4 * size_t(b);
        at[2 * j + 1] = slots + 4 * size_t(b) + 1;
        if (b < grid) n = 2 * j + 2;
      }
      ok = await(at, n, step, A.polls, got);
#pragma unroll
      for (int j = 0; j < 2 * kSlotsEach; j++)
        if (j < n) s[j & 1] += got[j];
    }
    warp_allsum(s);
    ok = __all_sync(kFull, ok);
    if (lane == 0) {
      sh.sum[0] = s[0];
      sh.sum[1] = s[1];
      if (!ok) sh.gave_up = 1;
    }
  } else {
    meanwhile();
  }
  __syncthreads();
  v[0] = sh.sum[0];
  v[1] = sh.sum[1];
  return sh.gave_up == 0;
}

// Shares of about the same number of blocks of S; the distinct cameras of a share's columns.
template <class W>
__global__ void __launch_bounds__(256) k_pcg_plan(W w) {
  __shared__ PcgSlot<W> slot;
  uint32_t bid, grid;
  const PcgSystem& A = block_system(w, slot, bid, grid);
  extern __shared__ uint32_t place[];  // C: 1 for a camera that occurs, then its place
  __shared__ uint32_t range[2], warp_sum[8];
  if (threadIdx.x < 2) {
    const uint64_t target = uint64_t(A.row_ptr[A.C]) * (bid + threadIdx.x) / grid;
    uint32_t lo = 0, hi = A.C;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) / 2;
      if (A.row_ptr[mid] < target) lo = mid + 1;
      else hi = mid;
    }
    range[threadIdx.x] = lo;
    A.share[bid + threadIdx.x] = lo;
  }
  for (uint32_t c = threadIdx.x; c < A.C; c += blockDim.x) place[c] = 0;
  __syncthreads();
  const uint32_t k0 = A.row_ptr[range[0]], k1 = A.row_ptr[range[1]];
  for (uint32_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) place[A.col[k]] = 1;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t base = 0;
  for (uint32_t c0 = 0; c0 < A.C; c0 += blockDim.x) {
    const uint32_t c = c0 + threadIdx.x;
    const bool on = c < A.C && place[c] != 0;
    const unsigned mask = __ballot_sync(kFull, on);
    if (lane == 0) warp_sum[warp] = __popc(mask);
    __syncthreads();
    uint32_t at = base;
    for (int w = 0; w < 8; w++) {
      if (w < warp) at += warp_sum[w];
      base += warp_sum[w];
    }
    at += __popc(mask & ((1u << lane) - 1u));
    if (on) {
      A.uni[size_t(bid) * A.C + at] = c;
      place[c] = at;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) A.uni_n[bid] = base;
  for (uint32_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) A.local[k] = place[A.col[k]];
}

// WIDE: for systems whose shares lie in global memory, 16-byte loads of S with two rows a lane: 25 -> 22 us a
// step at 1,500 cameras with the focal unknown, S in the L2.  From shared memory a row a lane is the faster
// one (a step at 7 cameras 2.6 and 3.5 us, at 61 cameras 5.8 and 7.0): its step is the instructions' latency.
template <bool SHARED, class W, bool WIDE = false>
__global__ void __launch_bounds__(kThreads, 1) k_pcg(W system, uint32_t limit) {
  after_previous();
  extern __shared__ __align__(16) double pcg_smem[];
  __shared__ Shared sh;
  __shared__ PcgSlot<W> slot;
  uint32_t bid, grid;
  const PcgSystem& A = block_system(system, slot, bid, grid);
  double* st = A.state;
  if (st[A.rhs ? A.solving : A.active] == 0 || limit == 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool alone = grid == 1;
  const uint32_t c0 = A.share[bid], c1 = A.share[bid + 1], nr = c1 - c0, rows = 6 * nr, first = 6 * c0, n = 6 * A.C;
  const uint32_t* uni = A.uni + size_t(bid) * A.C;
  const uint32_t cols = 6 * A.uni_n[bid];
  const uint32_t k0 = A.row_ptr[c0], blocks = A.row_ptr[c1] - k0;
  // Shared memory, as far as it goes: the direction and the columns' z, the own vectors, the rows' first
  // blocks, the own rows of S, their columns' places and the own preconditioner blocks.
  uint32_t used = 0;
  auto take = [&](size_t words, double* global) {
    if ((used + words) * sizeof(double) > kSmemBytes) return global;
    double* p = pcg_smem + used;
    used += uint32_t((words + 1) & ~size_t(1));
    return p;
  };
  double* pl = take(cols, A.pbuf + 2 * size_t(bid) * n);
  double* zl = alone ? nullptr : take(cols, A.pbuf + (2 * size_t(bid) + 1) * n);  // the columns' z of the next step
  double* own = take(4 * size_t(rows), nullptr);  // x, r, S p, z
  const bool keep = own != nullptr;
  double* xs = keep ? own : A.x + first;
  double* rs = keep ? own + rows : A.r + first;
  double* ss = keep ? own + 2 * size_t(rows) : A.p + first;  // p's place: the first direction is z
  double* zs = keep ? own + 3 * size_t(rows) : A.z + first;
  const uint32_t* row_ptr = A.row_ptr + c0;
  if (double* to = take((size_t(nr) + 2) / 2, nullptr)) {
    uint32_t* words = reinterpret_cast<uint32_t*>(to);
    for (uint32_t k = threadIdx.x; k <= nr; k += kThreads) words[k] = row_ptr[k];
    row_ptr = words;
  }
  // A block of S takes 38 words in shared memory, so that a warp's reads of five blocks fall on different
  // banks (36 where only they fit).  Eight iterations at 36 and 38 words, ms: 24 cameras 1.44 and 1.42, every
  // camera seeing every point 1.29 and 1.23, with the focal unknown 1.15 and 1.10; 61 cameras 2.34 and 2.29; a
  // batch of 24 windows 2.38 and 2.21, with the focal unknown 2.46 and 2.31; 7 and 10 cameras alike.
  const double* S = A.S + 36 * size_t(k0);
  const size_t rest = (size_t(blocks) + 1) / 2 + 36 * size_t(nr) + 4;  // the places and preconditioner blocks
  const uint32_t stride = (used + 38 * size_t(blocks) + rest) * sizeof(double) <= kSmemBytes ? 38 : 36;
  double* const staged = take(stride * size_t(blocks), nullptr);
  if (staged) {
    const double2* from = reinterpret_cast<const double2*>(S);
    for (uint32_t k = threadIdx.x; k < 18 * blocks; k += kThreads) {
      const uint32_t b = k / 18;
      reinterpret_cast<double2*>(staged)[stride / 2 * b + (k - 18 * b)] = from[k];
    }
    S = staged;
  }
  const uint32_t block_words = staged ? stride : 36;
  const uint32_t* local = A.local + k0;
  if (double* to = take((size_t(blocks) + 1) / 2, nullptr)) {
    uint32_t* words = reinterpret_cast<uint32_t*>(to);
    for (uint32_t k = threadIdx.x; k < blocks; k += kThreads) words[k] = local[k];
    local = words;
  }
  const double* Minv = A.Minv + 36 * size_t(c0);
  if (double* to = take(36 * size_t(nr), nullptr)) {
    for (uint32_t k = threadIdx.x; k < 36 * nr; k += kThreads) to[k] = Minv[k];
    Minv = to;
  }
  const bool starting = A.rhs != nullptr;
  for (uint32_t j = threadIdx.x; j < cols; j += kThreads) {
    const uint32_t b = j / 6;
    pl[j] = 0;  // (beta is zero in the first step)
    if (!alone && !starting) zl[j] = A.z[6 * uni[b] + (j - 6 * b)];
  }
  if (keep || starting)
    for (uint32_t i = threadIdx.x; i < rows; i += kThreads) {
      xs[i] = starting ? 0 : A.x[first + i];
      rs[i] = starting ? A.rhs[first + i] : A.r[first + i];
      if (!starting) zs[i] = A.z[first + i];
    }
  double xf = 0, rf = 0, zf = 0, pf = 0, sff = 0, finv = 0;  // the focal unknown, alike in every block
  if (SHARED && !starting) {
    xf = A.x[n];
    rf = A.r[n];
    zf = A.z[n];
    sff = st[A.focal_diag];
    finv = st[A.focal_inv];
  }
  double rho = st[A.rho], beta = 0, r0 = st[A.r0], r2 = st[A.r2];
  double inner = A.inner_r0 >= 0 ? st[A.inner_r0] : 0.0;
  // A warp per camera row, or several warps on a row's blocks; a lane sums one of the six rows over every
  // fifth block (WIDE: two rows over every tenth).  The first `owners` warps hold the own rows' scalars.
  const uint32_t splits = nr == 0 || nr >= uint32_t(kWarps) ? 1 : kWarps / nr;
  const int owners = int(min(uint32_t(kWarps), (rows + 31) / 32));
  const uint32_t lane_row = lane % 6, lane_block = lane / 6;
  bool active = true, failed = false, converged = false, ok = true;
  uint32_t it = 0;
  if (threadIdx.x == 0) sh.gave_up = 0;
  __syncthreads();
  // Index of own scalar row i in pl (a row's own camera is among its columns).
  auto place_of = [&](uint32_t i) {
    const uint32_t c = c0 + i / 6;
    uint32_t lo = 0, hi = cols / 6 - 1;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) / 2;
      if (uni[mid] < c) lo = mid + 1;
      else hi = mid;
    }
    return 6 * lo + i % 6;
  };
  const uint32_t my_place = threadIdx.x < rows ? place_of(threadIdx.x) : 0;
  const uint32_t my_part = threadIdx.x / 6 * splits, my_row = threadIdx.x % 6;
  const double* const znext = alone ? zs : zl;
  // z = M^-1 r of the own cameras (to the other blocks as the z of `step`); r . r and z . r.
  auto precondition = [&](uint64_t step, double (&v)[2]) {
    v[0] = v[1] = 0;
    for (uint32_t i = threadIdx.x; i < rows; i += kThreads) {
      const double* Mi = Minv + 6 * size_t(i);
      const double* rc = rs + i - i % 6;
      const double rr = rs[i];
      const double zz = (Mi[0] * rc[0] + Mi[1] * rc[1]) + (Mi[2] * rc[2] + Mi[3] * rc[3]) + (Mi[4] * rc[4] + Mi[5] * rc[5]);
      if (alone) zs[i] = zz;
      else publish(A.zx + first + i, zz, step);
      v[0] += rr * rr;
      v[1] += zz * rr;
    }
  };
  // The columns' z of `step`, while the first warp waits for the sums.
  auto fetch = [&](uint64_t step) {
    for (uint32_t j = threadIdx.x - 32; j < cols; j += 2 * (kThreads - 32)) {
      const uint32_t j1 = j + (kThreads - 32), b = j / 6, b1 = j1 / 6;
      const Flagged* at[2] = {A.zx + 6 * uni[b] + (j - 6 * b), nullptr};
      if (j1 < cols) at[1] = A.zx + 6 * uni[b1] + (j1 - 6 * b1);
      double got[2];
      if (*(volatile int*)&sh.gave_up != 0 || !await(at, j1 < cols ? 2 : 1, step, A.polls, got)) {
        *(volatile int*)&sh.gave_up = 1;
        break;
      }
      zl[j] = got[0];
      if (j1 < cols) zl[j1] = got[1];
    }
  };
  if (starting) {
    double focal = 0, full = 0;
    if (SHARED) {
      // H_ff and b_f with the points' shares, alike in every block.
      double t[4] = {0, 0, 0, 0};
      for (uint32_t b = threadIdx.x; b < A.scal_blocks; b += kThreads)
        for (int k = 0; k < 4; k++) t[k] += A.scal_part[4 * size_t(b) + k];
      warp_allsum(t);
      double* to = &sh.part[0][0];  // 16 x 6 values
      if (lane == 0)
        for (int k = 0; k < 4; k++) to[4 * warp + k] = t[k];
      __syncthreads();
      for (int k = 0; k < 4; k++) t[k] = 0;
      for (int w = 0; w < kWarps; w++)
        for (int k = 0; k < 4; k++) t[k] += to[4 * w + k];
      full = t[0] + st[A.lambda] * fmax(t[0], 1e-10);
      sff = full - t[2];
      finv = sff > 0 ? 1 / sff : -1;
      rf = focal = -t[1] - t[3];
      zf = finv * rf;
    }
    const bool fail = st[A.block_failed] != 0 || (SHARED && !(finv > 0));
    double v[2] = {0, 0};
    if (!fail) {
      precondition(1, v);
      ok = grid_sum(A, sh, v, 1, 1, owners, bid, grid, [&] { fetch(1); });
      r0 = r2 = inner = v[0] + rf * rf;
      rho = v[1] + rf * zf;
    }
    active = !fail && ok && r0 > 0 && rho > 0;
    if (bid == 0 && threadIdx.x == 0 && ok) {
      for (int k = A.clear_from; k <= A.clear_to; k++) st[k] = 0;
      if (SHARED) {
        st[A.focal_full] = full;
        st[A.focal_diag] = sff;
        st[A.focal_inv] = finv;
        st[A.focal_rhs] = focal;
      }
      if (!fail) {
        st[A.rho] = rho;
        st[A.r0] = st[A.r2] = st[A.inner_r0] = r0;
      }
      if (active) st[A.active] = 1;
      else if (fail || r0 > 1e-24) st[A.failed] = 1;
    }
    if (!active && ok) {
      // (x of a solve that starts at its solution is zero)
      if (!fail)
        for (uint32_t i = threadIdx.x; i < rows; i += kThreads) A.x[first + i] = 0;
      if (SHARED && !fail && bid == 0 && threadIdx.x == 0) A.x[n] = 0;
      return;
    }
  }
  const double bound = fmax(A.tol * A.tol * r0, A.inner_r0 >= 0 ? A.tol_inner * A.tol_inner * inner : 0.0);
  while (active && it < limit) {
    const uint64_t step = it + 2;
    for (uint32_t j = threadIdx.x; j < cols; j += kThreads) pl[j] = znext[j] + beta * pl[j];
    __syncthreads();
    for (uint32_t item = warp; item < nr * splits; item += kWarps) {
      const uint32_t row = splits == 1 ? item : item / splits, part = item - row * splits;
      const uint32_t b0 = row_ptr[row] - k0, nb = row_ptr[row + 1] - k0 - b0;
      const uint32_t lo = b0 + nb * part / splits, hi = b0 + nb * (part + 1) / splits;
      double* const out = splits == 1 ? ss + 6 * row : sh.part[item];
      if constexpr (WIDE) {
        double acc[2][2] = {{0, 0}, {0, 0}};
        const uint32_t pair = 2 * (lane % 3);
        if (lane < 30) {
#pragma unroll 2
          for (uint32_t b = lo + lane / 3; b < hi; b += 10) {
            const double2* Sb = reinterpret_cast<const double2*>(S + block_words * size_t(b) + pair);
            const double2* pb = reinterpret_cast<const double2*>(pl + 6 * local[b]);
#pragma unroll
            for (int k = 0; k < 3; k++) {
              const double2 pv = pb[k], s0 = Sb[6 * k], s1 = Sb[6 * k + 3];
              acc[0][0] += s0.x * pv.x;
              acc[0][1] += s0.y * pv.x;
              acc[1][0] += s1.x * pv.y;
              acc[1][1] += s1.y * pv.y;
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
          double a = acc[0][j] + acc[1][j];
          a += __shfl_down_sync(kFull, a, 15);
          const double b1 = __shfl_down_sync(kFull, a, 3), b2 = __shfl_down_sync(kFull, a, 6),
                       b3 = __shfl_down_sync(kFull, a, 9), b4 = __shfl_down_sync(kFull, a, 12);
          if (lane < 3) out[pair + j] = (a + b1) + (b2 + b3) + b4;
        }
      } else {
        double acc[3] = {0, 0, 0};  // independent sums: one chain of dependent FMAs a lane was half of a step
        if (lane < 30) {
#pragma unroll 2
          for (uint32_t b = lo + lane_block; b < hi; b += 5) {
            const double* Sb = S + block_words * size_t(b) + lane_row;
            const double2* pb = reinterpret_cast<const double2*>(pl + 6 * local[b]);
#pragma unroll
            for (int k = 0; k < 3; k++) {
              const double2 pv = pb[k];
              acc[2 * k % 3] += Sb[12 * k] * pv.x;
              acc[(2 * k + 1) % 3] += Sb[12 * k + 6] * pv.y;
            }
          }
        }
        acc[0] += acc[1] + acc[2];
        const double far = __shfl_down_sync(kFull, acc[0], 24), near = __shfl_down_sync(kFull, acc[0], 6),
                     mid = __shfl_down_sync(kFull, acc[0], 12), mid2 = __shfl_down_sync(kFull, acc[0], 18);
        if (lane < 6) {
          out[lane] = (acc[0] + near) + (mid + mid2) + far;
        }
      }
    }
    __syncthreads();
    if (SHARED) pf = zf + beta * pf;
    double v[2] = {0, 0};  // p . S p over the own camera rows, the focal row's camera share
    for (uint32_t i = threadIdx.x; i < rows; i += kThreads) {
      double sp = 0;
      if (splits == 1) {
        sp = ss[i];
      } else {  // (several warps a row: at most 15 rows of cameras, one scalar row a thread)
        for (uint32_t k = 0; k < splits; k++) sp += sh.part[my_part + k][my_row];
      }
      const double pv = pl[i == threadIdx.x ? my_place : place_of(i)];
      if (SHARED) {
        const double f = A.scf[first + i];
        sp += f * pf;
        v[1] += f * pv;
      }
      ss[i] = sp;
      v[0] += pv * sp;
    }
    if (!(ok = grid_sum(A, sh, v, step, 0, owners, bid, grid, [] {}))) break;
    const double spf = SHARED ? sff * pf + v[1] : 0.0, den = SHARED ? v[0] + pf * spf : v[0], alpha = rho / den;
    if (!(den > 0) || !(fabs(alpha) < A.alpha_limit)) {
      active = false;
      failed = true;
      break;
    }
    for (uint32_t i = threadIdx.x; i < rows; i += kThreads) {
      xs[i] += alpha * pl[i == threadIdx.x ? my_place : place_of(i)];
      rs[i] -= alpha * ss[i];
    }
    __syncthreads();
    precondition(step, v);
    if (!(ok = grid_sum(A, sh, v, step, 1, owners, bid, grid, [&] { fetch(step); }))) break;
    it++;
    r2 = v[0];
    double next = v[1];
    if (SHARED) {
      xf += alpha * pf;
      rf -= alpha * spf;
      zf = finv * rf;
      r2 += rf * rf;
      next += rf * zf;
    }
    if (r2 <= bound) {
      active = false;
      converged = true;
    } else if (!(next > 0)) {
      active = false;
      failed = true;
    } else {
      beta = next / rho;
      rho = next;
    }
  }
  if (keep)
    for (uint32_t i = threadIdx.x; i < rows; i += kThreads) {
      A.x[first + i] = xs[i];
      A.r[first + i] = rs[i];
    }
  if (threadIdx.x != 0 || (bid != 0 && ok)) return;
  if (!ok) {
    st[A.wait] = 1;
    st[A.failed] = 1;
    st[A.active] = 0;
    return;
  }
  if (SHARED) {
    A.x[n] = xf;
    A.r[n] = rf;
  }
  st[A.steps] += it;
  if (A.all_steps >= 0) st[A.all_steps] += it;
  st[A.r2] = r2;
  st[A.rho] = rho;
  if (failed) st[A.failed] = 1;
  if (converged && A.converged >= 0) st[A.converged] = 1;
  if (!active) st[A.active] = 0;
}

}  // namespace

cudaError_t pcg_configure() {
  const void* kernels[] = {
      reinterpret_cast<const void*>(k_pcg<false, PcgSystem>), reinterpret_cast<const void*>(k_pcg<true, PcgSystem>),
      reinterpret_cast<const void*>(k_pcg<false, PcgSystem, true>), reinterpret_cast<const void*>(k_pcg<true, PcgSystem, true>),
      reinterpret_cast<const void*>(k_pcg<false, PcgMany>), reinterpret_cast<const void*>(k_pcg<true, PcgMany>)};
  for (const void* f : kernels) {
    const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemBytes));
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

uint32_t pcg_grid(uint64_t blocks, uint32_t C, int sms) {
  const uint64_t bytes = 288 * blocks;
  if (bytes + (5 * 6 + 36) * 8 * uint64_t(C) <= kSmemBytes) return 1;  // all in one block: nothing to exchange
  const uint64_t share = 48 * 1024;
  return uint32_t(std::min<uint64_t>(std::min<uint64_t>((bytes + share - 1) / share, C), uint64_t(std::max(1, sms))));
}

uint32_t pcg_launch_plan(const PcgSystem& a, uint32_t grid, cudaStream_t s) {
  k_pcg_plan<PcgSystem><<<grid, 256, size_t(a.C) * sizeof(uint32_t), s>>>(a);
  return 1;
}

cudaError_t launch_pcg(const PcgSystem& a, uint32_t limit, uint32_t grid, cudaStream_t s) {
  auto f = a.shared ? k_pcg<true, PcgSystem> : k_pcg<false, PcgSystem>;
  // Where the shares cannot all lie in shared memory.
  if (288 * uint64_t(a.max_blocks) > uint64_t(grid) * kSmemBytes)
    f = a.shared ? k_pcg<true, PcgSystem, true> : k_pcg<false, PcgSystem, true>;
  if (grid == 1) return launch_dependent(f, 1, kThreads, kSmemBytes, s, a, limit);
  // No step of an earlier run may be taken for one of this run's.
  cudaError_t e = cudaMemsetAsync(a.zx, 0, 6 * size_t(a.C) * sizeof(Flagged), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(a.slots, 0, 4 * size_t(grid) * sizeof(Flagged), s);
  if (e != cudaSuccess) return e;
  PcgSystem q = a;
  void* args[] = {&q, &limit};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(f), dim3(grid), dim3(kThreads), args, kSmemBytes, s);
}

uint32_t pcg_launch_many_plan(const PcgMany& b, uint32_t count, uint32_t max_cameras, cudaStream_t s) {
  k_pcg_plan<PcgMany><<<count, 256, size_t(max_cameras) * sizeof(uint32_t), s>>>(b);
  return 1;
}

cudaError_t launch_many_pcg(const PcgMany& b, uint32_t count, bool shared, uint32_t limit, cudaStream_t s) {
  const auto f = shared ? k_pcg<true, PcgMany> : k_pcg<false, PcgMany>;
  f<<<count, kThreads, kSmemBytes, s>>>(b, limit);
  return cudaGetLastError();
}

}  // namespace tba
