// Device-side structural checks of a packed problem; see tba_checks.cuh.  Every kernel records the
// smallest failing position of its check with an atomic minimum, so the host can report the
// failure a serial scan in the same order would meet first.
#include "tba_checks.cuh"

#include "tba_launch.cuh"

namespace tba {
namespace {

__global__ void __launch_bounds__(256) k_check_points(CheckParams A) {
  after_previous();
  const uint32_t* ps = A.index + 2 * size_t(A.M);
  const uint32_t* obs_point = A.index + A.M;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < A.P; p += gridDim.x * blockDim.x) {
    const uint32_t b = ps[p], e = ps[p + 1];
    unsigned long long key = ~0ull;
    if (e > A.M) {
      key = (uint64_t(p) << 2) | 0;
    } else if (uint64_t(e) < uint64_t(b) + 2) {
      key = (uint64_t(p) << 2) | 1;
    } else {
      for (uint32_t i = b; i < e; i++)
        if (obs_point[i] != p) {
          key = (uint64_t(p) << 2) | 2;
          break;
        }
    }
    if (key != ~0ull) atomicMin(A.keys + CK_POINTS, key);
  }
}

__global__ void __launch_bounds__(256) k_check_cameras(CheckParams A) {
  after_previous();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < A.M; i += gridDim.x * blockDim.x)
    if (A.index[i] >= A.C) atomicMin(A.keys + CK_CAMERA, (unsigned long long)i);
}

// One block per camera (grid-stride): every entry of the camera's list must be an observation of
// that camera, claimed once.  The camera offsets were checked on the host (monotone, within M).
__global__ void __launch_bounds__(256) k_check_lists(CheckParams A) {
  after_previous();
  const uint32_t* obs_camera = A.index;
  const uint32_t* cs = A.index + 2 * size_t(A.M) + A.P + 1;
  const uint32_t* cam_obs = cs + A.C + 1;
  for (uint32_t cam = blockIdx.x; cam < A.C; cam += gridDim.x) {
    bool bad = false;
    for (uint32_t k = cs[cam] + threadIdx.x; k < cs[cam + 1]; k += blockDim.x) {
      const uint32_t i = cam_obs[k];
      if (i >= A.M || obs_camera[i] != cam || atomicAdd(A.claims + i, 1u) != 0) bad = true;
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicMin(A.keys + CK_LISTS, (unsigned long long)cam);
  }
}

__global__ void __launch_bounds__(256) k_check_scene(const double* x, uint64_t n, uint64_t base,
                                                      unsigned long long* keys) {
  after_previous();
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
    const double v = x[i];
    if (!isfinite(v) || fabs(v) > 1e9 || (v != 0 && fabs(v) < 1e-30))
      atomicMin(keys + CK_SCENE, (unsigned long long)(base + i));
  }
}

__device__ inline bool outside(double v) { return !isfinite(v) || fabs(v) > 1e9 || (v != 0 && fabs(v) < 1e-30); }

// Every check of a problem, strided over its blocks.  The host has checked the camera offsets.
__global__ void __launch_bounds__(256) k_check_batch(const CheckProblem* problems, const uint2* work, uint32_t* bad) {
  const uint2 w = work[blockIdx.x];
  const CheckProblem A = problems[w.x];
  const uint32_t first = w.y * blockDim.x + threadIdx.x, step = A.blocks * blockDim.x;
  const uint32_t* obs_camera = A.index;
  const uint32_t* obs_point = A.index + A.M;
  const uint32_t* ps = obs_point + A.M;
  const uint32_t* cs = ps + A.P + 1;
  const uint32_t* cam_obs = cs + A.C + 1;
  bool failed = false;
  for (uint32_t p = first; p < A.P; p += step) {
    const uint32_t b = ps[p], e = ps[p + 1];
    if (e > A.M || uint64_t(e) < uint64_t(b) + 2) {
      failed = true;
    } else {
      for (uint32_t i = b; i < e; i++) failed = failed || obs_point[i] != p;
    }
  }
  for (uint32_t i = first; i < A.M; i += step) failed = failed || obs_camera[i] >= A.C;
  for (uint32_t cam = w.y; cam < A.C; cam += A.blocks)
    for (uint32_t k = cs[cam] + threadIdx.x; k < cs[cam + 1]; k += blockDim.x) {
      const uint32_t i = cam_obs[k];
      if (i >= A.M || obs_camera[i] != cam || atomicAdd(A.claims + i, 1u) != 0) failed = true;
    }
  const uint64_t n = 18ull * A.C + 3ull * A.P + 2ull * A.M;
  for (uint64_t i = first; i < n; i += step) failed = failed || outside(A.scene[i]);
  if (__syncthreads_or(failed) && threadIdx.x == 0) *bad = 1;
}

__global__ void __launch_bounds__(256) k_check_observations(ObservationChecks A) {
  const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  bool failed = false;
  const uint2* ix = reinterpret_cast<const uint2*>(A.indices);
  // An observation lies in the track of its point: with offsets that never decrease and cover the
  // observations, that is every track's observations being its point's.  (A thread a track took 12 ms for two
  // tracks of 200,000 observations, each load waiting for the one before; this is one pass.)
  for (uint64_t i = first; i < A.M; i += step) {
    const uint2 v = ix[i];
    if (v.x >= A.C || v.y >= A.P) failed = true;
    else if (A.offsets) failed = failed || i < A.offsets[v.y] || i >= A.offsets[v.y + 1];
  }
  if (A.offsets)
    for (uint64_t h = first; h < A.P; h += step) {
      const uint32_t b = A.offsets[h], e = A.offsets[h + 1];
      failed = failed || e < b || e > A.M;
    }
  for (int k = 0; k < 3; k++)
    for (uint64_t i = first; i < A.counts[k]; i += step) failed = failed || outside(A.values[k][i]);
  if (__syncthreads_or(failed) && threadIdx.x == 0) *A.bad = 1;
}

}  // namespace

void launch_check_batch(const CheckProblem* problems, const uint2* work, uint32_t blocks, uint32_t* bad, cudaStream_t s) {
  k_check_batch<<<blocks, 256, 0, s>>>(problems, work, bad);
}

void launch_check_observations(const ObservationChecks& p, int sms, cudaStream_t s) {
  const uint64_t most = p.M > p.P ? p.M : p.P;
  const uint64_t want = (most + 255) / 256, cap = 8ull * uint64_t(sms > 0 ? sms : 1);
  k_check_observations<<<uint32_t(want < 1 ? 1 : (want < cap ? want : cap)), 256, 0, s>>>(p);
}

cudaError_t launch_checks(const CheckParams& p, int sms, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(p.keys, 0xff, CK_WORDS * sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  const uint32_t grid = uint32_t(sms > 0 ? sms : 1) * 8;
  if (p.P) launch_dependent(k_check_points, grid, 256, 0, s, p);
  if (p.M) launch_dependent(k_check_cameras, grid, 256, 0, s, p);
  if (p.lists && p.C) {
    if (p.M) {
      e = cudaMemsetAsync(p.claims, 0, sizeof(uint32_t) * p.M, s);
      if (e != cudaSuccess) return e;
    }
    launch_dependent(k_check_lists, p.C < 4u * uint32_t(sms) ? p.C : 4u * uint32_t(sms), 256, 0, s, p);
  }
  for (int k = 0; k < 4; k++)
    if (p.len[k]) launch_dependent(k_check_scene, grid, 256, 0, s, p.seg[k], p.len[k], p.base[k], p.keys);
  return cudaGetLastError();
}

}  // namespace tba
