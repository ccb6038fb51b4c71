// The C ABI of libtba.so (include/tba.h) and the host side of one solve: structural checks of
// the packed arrays, the warp-task and camera-chunk schedules, the device workspace, and the LM
// loop that enqueues the grid engine's kernels (tba_kernels.cu).
//
// The loop is the reference's plan (src/sfm/bundle/gpu/bundle.ts:314-772 and
// joint-focal.ts:330-880) with its host round trips reduced to one small read per PCG chunk and
// one per LM iteration: every kernel is guarded by the device state words, so an iteration past
// convergence is a no-op and the reads only end the loops early.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <numeric>
#include <string>
#include <thread>
#include <vector>

#include "../../include/tba.h"
#include "tba_adjoint.cuh"
#include "tba_batch.cuh"
#include "tba_engine.cuh"
#include "tba_checks.cuh"
#include "tba_observations.cuh"
#include "tba_pcg.cuh"
#include "tba_schur.cuh"

using tba::Params;

// The device-side PCG loop of one product form: a graph of one while node whose body is a PCG
// step (product, column sums and alpha, x/r/z update and beta, new direction) and k_pcg_loop_next,
// which counts the step and ends the loop when the PCG stops or its budget is spent.  The graph
// bakes the launch parameters; `key` holds them, and a solve with the same parameters (the same
// scene shape in the same workspace) launches it again instead of building a new one.
struct PcgLoop {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  std::vector<char> key;
  uint32_t body_kernels = 0;  // kernels of one body iteration
  void release() {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    exec = nullptr;
    graph = nullptr;
    key.clear();
  }
};

struct tba_device {
  int ordinal = 0;
  int sms = 0;
  cudaStream_t stream = nullptr;
  cudaStream_t down = nullptr;  // device-to-host copies that overlap the next slice's upload and kernel
  std::mutex mu;
  std::string error;
  char* arena = nullptr;
  size_t capacity = 0;
  // The explicit reduced camera system's structure and blocks (grown as needed, like the arena).
  char* schur = nullptr;
  size_t schur_capacity = 0;
  double* pinned = nullptr;  // small host buffer for flag reads
  std::vector<cudaEvent_t> events;
  // Polls of each main-loop wait of the inverse-depth linearisation and, up to its own bound, of each wait
  // between the blocks of a PCG (tba_device_set_wait_limit).
  uint32_t wait_limit = tba::kIdWaitPolls;
  uint32_t pcg_polls() const { return std::min(wait_limit, tba::kPcgWaitPolls); }
  // Batched solves: their own workspace, the cached graph of the last launch and its key, and
  // the autotuner's choices by batch shape.
  char* batch_arena = nullptr;
  size_t batch_capacity = 0;
  cudaGraphExec_t batch_graph = nullptr;
  std::vector<char> batch_key;
  // One LM iteration of a batch on the grid kernels.
  cudaGraphExec_t window_graph = nullptr;
  std::vector<char> window_key;
  std::map<std::string, int> tuned;
  // The grid engine's device-side PCG loops (the solve's own product and the mixed form's FP64
  // tail) and the adjoint's.
  PcgLoop pcg_loops[2];
  PcgLoop adj_loop;
  // Set when the driver could not build a conditional graph: the PCG steps then run from the host.
  bool host_pcg_only = false;
};

// A scene resident on the device between calls: the packed arrays of one problem and its host
// schedules.
struct tba_scene {
  tba_device* device = nullptr;
  tba_control shape{};
  double* scene = nullptr;     // device, tba_scene_size doubles
  uint32_t* index = nullptr;   // device, tba_index_size words
  void* plan = nullptr;        // HostPlan
  uint32_t* plan_dev = nullptr;  // device copy of the plan's arrays (HostPlan::sections order)
};

namespace {

std::string g_open_error;

struct Fail {
  tba_status status;
  std::string message;
};

#define CUDA_TRY(expr)                                                                     \
  do {                                                                                     \
    cudaError_t _e = (expr);                                                               \
    if (_e != cudaSuccess)                                                                 \
      throw Fail{TBA_ERROR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(_e)};      \
  } while (0)

[[noreturn]] void argument(const std::string& m) { throw Fail{TBA_ERROR_ARGUMENT, m}; }

// A bump allocator over the device workspace (256-byte aligned sections).
struct Layout {
  size_t bytes = 0;
  template <typename T>
  size_t take(size_t count) {
    const size_t at = bytes;
    bytes += (count * sizeof(T) + 255) / 256 * 256;
    return at;
  }
};

// bundleProblem's option limits (src/sfm/bundle/gpu/bundle-host.ts:49-65) and the gauge and
// window rules it checks (:66-96), on the packed control block.
void check_control(const tba_control* c) {
  if (!c) argument("Invalid GPU BA scene/options: no control block");
  if (c->cameras < 2 || c->points < 1 || c->directional_points >= c->points + 0u ||
      c->iterations > 100 || !(std::isfinite(c->huber) && c->huber >= 1e-12 && c->huber <= 1e6) ||
      c->max_cg < 1 || c->max_cg > 256 ||
      !(std::isfinite(c->cg_tolerance) && c->cg_tolerance >= 1e-12 && c->cg_tolerance <= 1e-2) ||
      !(std::isfinite(c->stall_tolerance) && c->stall_tolerance >= 0 && c->stall_tolerance < 1) ||
      c->precision > 1 ||
      (c->flags & ~(TBA_FLAG_TIME_PRODUCTS | TBA_FLAG_PRODUCT_ERROR | TBA_FLAG_HOST_PCG_LOOP)) != 0)
    argument("Invalid GPU BA scene/options");
  if (c->anchor >= c->cameras || c->scale_view >= c->cameras || c->anchor == c->scale_view)
    argument("Invalid GPU BA gauge cameras");
}

// The structure of the packed index array (bundleIndexLayout): every section consistent with the
// others, so that no kernel can index out of bounds.
// Runs f(begin, end, worker) over [0, n) split into up to `threads` contiguous ranges on host
// threads (serially below `serial_below`).
template <typename F>
void parallel_ranges(uint64_t n, uint64_t serial_below, F f) {
  const unsigned threads = unsigned(std::min<uint64_t>(n, std::min(16u, std::max(1u, std::thread::hardware_concurrency()))));
  if (n < serial_below || threads <= 1) {
    f(uint64_t(0), n, 0u);
    return;
  }
  std::vector<std::thread> pool;
  for (unsigned t = 0; t < threads; t++)
    pool.emplace_back([&, t] { f(n * t / threads, n * (t + 1) / threads, t); });
  for (auto& th : pool) th.join();
}

// The first failure over parallel ranges: the lowest position that failed, and its message.
struct FirstFailure {
  std::mutex mu;
  uint64_t at = UINT64_MAX;
  const char* message = nullptr;
  void record(uint64_t where, const char* m) {
    std::lock_guard<std::mutex> lock(mu);
    if (where < at) {
      at = where;
      message = m;
    }
  }
  void raise() const {
    if (message) argument(message);
  }
};

// The structure of the packed index array (bundleIndexLayout): every section consistent with the
// others, so that no kernel can index out of bounds.  Large arrays are checked on host threads;
// the failure reported is the one a serial scan in this order would meet first.
void check_index(const tba_control* c, const uint32_t* index) {
  const uint64_t C = c->cameras, P = c->points, M = c->observations;
  const uint32_t* obs_camera = index;
  const uint32_t* obs_point = index + M;
  const uint32_t* ps = index + 2 * M;
  const uint32_t* cs = ps + P + 1;
  const uint32_t* cam_obs = cs + C + 1;
  const uint32_t* active = cam_obs + M;
  if (ps[0] != 0 || ps[P] != M) argument("Invalid GPU BA index: point offsets do not cover the observations");
  {
    FirstFailure ff;
    parallel_ranges(P, 1u << 16, [&](uint64_t b, uint64_t e, unsigned) {
      for (uint64_t p = b; p < e; p++) {
        if (ps[p + 1] > M) return ff.record(p, "Invalid GPU BA index: point offsets exceed the observations");
        if (ps[p + 1] < ps[p] + 2) return ff.record(p, "Landmarks require at least two observations");
        for (uint64_t i = ps[p]; i < ps[p + 1]; i++)
          if (obs_point[i] != p)
            return ff.record(p, "Invalid GPU BA index: observation point does not match the point offsets");
      }
    });
    ff.raise();
  }
  {
    FirstFailure ff;
    parallel_ranges(M, 1u << 18, [&](uint64_t b, uint64_t e, unsigned) {
      for (uint64_t i = b; i < e; i++)
        if (obs_camera[i] >= C) return ff.record(i, "Invalid GPU BA index: observation camera out of range");
    });
    ff.raise();
  }
  if (cs[0] != 0 || cs[C] != M) argument("Invalid GPU BA index: camera offsets do not cover the observations");
  for (uint64_t cam = 0; cam < C; cam++)
    if (cs[cam + 1] < cs[cam] || cs[cam + 1] > M)
      argument("Invalid GPU BA index: camera offsets decrease or exceed the observations");
  {
    // Each observation may be claimed only by its own camera, so a thread owning a range of
    // cameras is the only one to touch `seen` for their observations.
    std::vector<uint8_t> seen(M, 0);
    FirstFailure ff;
    parallel_ranges(C, M < (1u << 18) ? C + 1 : 1, [&](uint64_t b, uint64_t e, unsigned) {
      for (uint64_t cam = b; cam < e; cam++)
        for (uint64_t k = cs[cam]; k < cs[cam + 1]; k++) {
          const uint32_t i = cam_obs[k];
          if (i >= M || obs_camera[i] != cam || seen[i])
            return ff.record(cam, "Invalid GPU BA index: camera observation lists are not the observations of each camera");
          seen[i] = 1;
        }
    });
    ff.raise();
  }
  uint32_t fixed = 0;
  for (uint64_t cam = 0; cam < C; cam++) {
    if (active[cam] > 1) argument("Invalid GPU BA index: camera activity flags must be 0 or 1");
    fixed += active[cam] == 0;
  }
  if (active[c->anchor] != 0) argument("Invalid GPU BA gauge cameras: the anchor must be fixed");
  if (fixed > 1 && active[c->scale_view] != 0) argument("Local GPU BA scale camera must be fixed");
}

// finiteGpuArray and validateGpuCamera (src/geometry/gpu/bounds.ts:5-26) on the scene array.
void check_scene(const tba_control* c, const double* scene, size_t len) {
  FirstFailure ff;
  parallel_ranges(len, 1u << 18, [&](uint64_t b, uint64_t e, unsigned) {
    for (uint64_t i = b; i < e; i++) {
      const double x = scene[i];
      if (!std::isfinite(x) || std::fabs(x) > 1e9 || (x != 0 && std::fabs(x) < 1e-30))
        return ff.record(i, "GPU BA input exceeds supported coordinate bounds");
    }
  });
  ff.raise();
  const double* k = scene + 12 * size_t(c->cameras) + 3 * size_t(c->points);
  for (uint32_t cam = 0; cam < c->cameras; cam++, k += 6)
    if (!(k[0] > 0 && k[1] > 0) || k[0] < 1e-6 || k[1] < 1e-6 || k[0] > 1e6 || k[1] > 1e6 ||
        std::max(std::fabs(k[2]), std::fabs(k[3])) > 1e9 || std::max(std::fabs(k[4]), std::fabs(k[5])) > 1)
      argument("Camera exceeds the supported GPU geometry bounds");
}

// The O(1) and O(C) parts of check_index and check_scene, on the host, with the message each would
// raise (null where it passes); the O(M) and O(P) parts run on the device after the upload
// (tba_checks.cu), and raise_checks reports the failure that check_index then check_scene, in
// their order, would meet first.
struct HostChecks {
  const char* point_ends = nullptr;     // before the per-point checks
  const char* camera_ends = nullptr;    // after the observation cameras
  const char* camera_offsets = nullptr;
  const char* activity = nullptr;       // after the camera lists
  const char* camera_bounds = nullptr;  // after the scene values
};

HostChecks host_checks(const tba_control* c, const uint32_t* index, const double* scene) {
  HostChecks h;
  const uint64_t C = c->cameras, P = c->points, M = c->observations;
  const uint32_t* ps = index + 2 * M;
  const uint32_t* cs = ps + P + 1;
  const uint32_t* active = cs + C + 1 + M;
  if (ps[0] != 0 || ps[P] != M) h.point_ends = "Invalid GPU BA index: point offsets do not cover the observations";
  if (cs[0] != 0 || cs[C] != M) h.camera_ends = "Invalid GPU BA index: camera offsets do not cover the observations";
  for (uint64_t cam = 0; cam < C && !h.camera_offsets; cam++)
    if (cs[cam + 1] < cs[cam] || cs[cam + 1] > M)
      h.camera_offsets = "Invalid GPU BA index: camera offsets decrease or exceed the observations";
  uint32_t fixed = 0;
  for (uint64_t cam = 0; cam < C && !h.activity; cam++) {
    if (active[cam] > 1) h.activity = "Invalid GPU BA index: camera activity flags must be 0 or 1";
    fixed += active[cam] == 0;
  }
  if (!h.activity && active[c->anchor] != 0) h.activity = "Invalid GPU BA gauge cameras: the anchor must be fixed";
  if (!h.activity && fixed > 1 && active[c->scale_view] != 0) h.activity = "Local GPU BA scale camera must be fixed";
  const double* k = scene + 12 * size_t(C) + 3 * size_t(P);
  for (uint64_t cam = 0; cam < C && !h.camera_bounds; cam++, k += 6)
    if (!(k[0] > 0 && k[1] > 0) || k[0] < 1e-6 || k[1] < 1e-6 || k[0] > 1e6 || k[1] > 1e6 ||
        std::max(std::fabs(k[2]), std::fabs(k[3])) > 1e9 || std::max(std::fabs(k[4]), std::fabs(k[5])) > 1)
      h.camera_bounds = "Camera exceeds the supported GPU geometry bounds";
  return h;
}

void raise_checks(const HostChecks& h, const unsigned long long* keys) {
  const unsigned long long none = ~0ull;
  if (h.point_ends) argument(h.point_ends);
  if (keys[tba::CK_POINTS] != none) {
    static const char* const messages[3] = {"Invalid GPU BA index: point offsets exceed the observations",
                                            "Landmarks require at least two observations",
                                            "Invalid GPU BA index: observation point does not match the point offsets"};
    argument(messages[keys[tba::CK_POINTS] & 3]);
  }
  if (keys[tba::CK_CAMERA] != none) argument("Invalid GPU BA index: observation camera out of range");
  if (h.camera_ends) argument(h.camera_ends);
  if (h.camera_offsets) argument(h.camera_offsets);
  if (keys[tba::CK_LISTS] != none)
    argument("Invalid GPU BA index: camera observation lists are not the observations of each camera");
  if (h.activity) argument(h.activity);
  if (keys[tba::CK_SCENE] != none) argument("GPU BA input exceeds supported coordinate bounds");
  if (h.camera_bounds) argument(h.camera_bounds);
}

// The adjoint, the observation evaluation and the batch on the grid kernels leave the O(M) checks to the
// device from this many observations on; below, the kernels' launches and the read cost more than the host's
// pass over the arrays.  Whole calls, checks on the host and on the device: an evaluation of 2,046
// observations 134 and 145 us, of 8,190 157 and 135, of 32,772 312 and 185, of 299,873 2,000 and 870; an
// adjoint 279 and 294, 376 and 362, 695 and 548, 3,300 and 1,840; a batch of two such windows 547 and 580,
// 653 and 630, 980 and 817 (32,772 each).
constexpr uint64_t kDeviceCheckMin = 8192;

// The device's part of the checks, on arrays just uploaded, and the first failure of both parts raised;
// `claims` is M words of scratch, `keys` CK_WORDS words.
void device_checks(tba_device* d, const HostChecks& h, uint32_t C, uint32_t P, uint32_t M, const uint32_t* index,
                   const double* const (&sections)[4], uint32_t* claims, unsigned long long* keys) {
  tba::CheckParams cp{};
  cp.C = C;
  cp.P = P;
  cp.M = M;
  cp.index = index;
  const uint64_t len[4] = {12 * uint64_t(C), 3 * uint64_t(P), 6 * uint64_t(C), 2 * uint64_t(M)};
  uint64_t base = 0;
  for (int k = 0; k < 4; k++) {
    cp.seg[k] = sections[k];
    cp.base[k] = base;
    cp.len[k] = len[k];
    base += len[k];
  }
  cp.claims = claims;
  cp.keys = keys;
  cp.lists = !h.camera_ends && !h.camera_offsets;
  CUDA_TRY(tba::launch_checks(cp, d->sms, d->stream));
  CUDA_TRY(cudaMemcpyAsync(d->pinned, keys, tba::CK_WORDS * sizeof(unsigned long long), cudaMemcpyDeviceToHost, d->stream));
  CUDA_TRY(cudaStreamSynchronize(d->stream));
  unsigned long long found[tba::CK_WORDS];
  std::memcpy(found, d->pinned, sizeof found);
  raise_checks(h, found);
}

// Runs of whole points of at most 32 observations; a longer point is a run of its own.
std::vector<uint32_t> build_tasks(const uint32_t* ps, uint32_t P) {
  std::vector<uint32_t> tasks;
  tasks.reserve(P / 4 + 2);
  uint32_t p = 0;
  while (p < P) {
    tasks.push_back(p);
    uint32_t n = ps[p + 1] - ps[p];
    p++;
    if (n > uint32_t(tba::kTaskObs)) continue;
    while (p < P && n + (ps[p + 1] - ps[p]) <= uint32_t(tba::kTaskObs)) {
      n += ps[p + 1] - ps[p];
      p++;
    }
  }
  tasks.push_back(P);
  return tasks;
}

struct Chunks {
  std::vector<uint32_t> cam, beg, cam_first;
};

// Chunks of each camera's observation list, sized so that the camera pass has a few blocks per SM over
// M observations in all.
uint32_t chunk_size(uint64_t M, int sms) {
  const uint64_t size = M / uint64_t(std::max(1, 8 * sms));
  return uint32_t(std::min<uint64_t>(2048, std::max<uint64_t>(128, (size + 127) / 128 * 128)));
}

Chunks build_chunks(const uint32_t* cs, uint32_t C, uint32_t size) {
  Chunks ch;
  for (uint32_t c = 0; c < C; c++) {
    ch.cam_first.push_back(uint32_t(ch.cam.size()));
    const uint32_t n = cs[c + 1] - cs[c];
    const uint32_t k = std::max<uint32_t>(1, (n + size - 1) / size);
    for (uint32_t j = 0; j < k; j++) {
      ch.cam.push_back(c);
      ch.beg.push_back(cs[c] + uint32_t(uint64_t(n) * j / k));
    }
  }
  ch.cam_first.push_back(uint32_t(ch.cam.size()));
  ch.beg.push_back(cs[C]);
  return ch;
}

void check_waits(const double* words) {
  if (words[tba::S_WAIT] != 0) throw Fail{TBA_ERROR_CUDA, "GPU BA: a wait between the PCG's blocks ran out"};
}

// Reads the state words into the pinned buffer; returns word `word`.
double read_word(tba_device* d, const double* state, int word) {
  CUDA_TRY(cudaMemcpyAsync(d->pinned, state, tba::S_READ * sizeof(double), cudaMemcpyDeviceToHost, d->stream));
  CUDA_TRY(cudaStreamSynchronize(d->stream));
  check_waits(d->pinned);
  return d->pinned[word];
}

// ---- the explicit reduced camera system ------------------------------------------------------------

// 6x6 blocks of S at most.
uint64_t schur_block_bound(uint64_t C, uint64_t pairs) { return std::min(C * C, 2 * pairs + C); }

// Pairs of observations of one point (all cameras counted as variable), the longest track, and the blocks of S
// that its camera pairs spread over (0: not looked for).
struct Tracks {
  uint64_t pairs = 0;
  uint32_t longest = 0;
  double spread = 0;
};

Tracks count_pairs(const uint32_t* ps, uint32_t P) {
  uint64_t squares = 0, sum = 0;
  Tracks t;
  for (uint32_t p = 0; p < P; p++) {
    const uint32_t n = ps[p + 1] - ps[p];
    squares += uint64_t(n) * n;
    sum += n;
    t.longest = std::max(t.longest, n);
  }
  t.pairs = (squares - sum) / 2;
  return t;
}

constexpr double kFarSystem = 110e6;  // bytes of S beyond which a step no longer finds it in the L2

// How many blocks of S the camera pairs spread over as if evenly: K of them, one from each of K points all along
// the list, agree with one another about K^2 / 2D times when they are spread over D.  Where cameras share points
// with their neighbours D is below 46,000 (spheres of 331 to 4,000 cameras, helices of 1,000 and 3,000), where
// any camera meets any other it is all pairs: 165,000 at 600 cameras, 950,000 at 4,600.  Taken 256 at a time
// until they agree often enough to tell; 20 to 60 us, 130 with the arrays out of the caches.  (The arrays are not
// yet checked.)
double spread_blocks(uint32_t C, uint32_t P, uint32_t M, const uint32_t* index) {
  constexpr uint32_t kSamples = 2048, kStep = 256, kPlaces = 4096;
  const uint32_t* ps = index + 2 * size_t(M);
  const uint32_t samples = std::min(kSamples, P);
  // Golden-ratio steps along the list, so that any first few of them lie evenly.
  const auto point = [&](uint32_t k) { return uint32_t(uint64_t(P) * (k * 1265 % kSamples) / kSamples); };
  std::vector<uint64_t> key(kPlaces, UINT64_MAX);
  std::vector<uint32_t> met(kPlaces, 0), last(kPlaces, UINT32_MAX);
  uint32_t one[kStep], two[kStep], from[kStep];
  uint64_t sampled = 0, agreed = 0, random = 88172645463325252ull;
  double blocks = 0;
  for (uint32_t k0 = 0; k0 < samples; k0 += kStep) {
    const uint32_t take = std::min(kStep, samples - k0);
    for (uint32_t k = 0; k < take; k++) __builtin_prefetch(ps + point(k0 + k));
    for (uint32_t k = 0; k < take; k++) {
      const uint32_t p = point(k0 + k), b = ps[p], e = ps[p + 1];
      one[k] = two[k] = 0;
      from[k] = p;
      if (e > M || uint64_t(e) < uint64_t(b) + 2) continue;
      random = random * 6364136223846793005ull + 1442695040888963407ull;
      const uint32_t n = e - b, i = uint32_t((random >> 33) % n);
      one[k] = b + i;
      two[k] = b + (i + 1 + uint32_t((random >> 20) % (n - 1))) % n;
      __builtin_prefetch(index + one[k]);
      __builtin_prefetch(index + two[k]);
    }
    for (uint32_t k = 0; k < take; k++) {
      const uint32_t c = index[one[k]], d = index[two[k]];
      if (one[k] == two[k] || c == d) continue;
      const uint64_t pair = (uint64_t(std::min(c, d)) << 32) | std::max(c, d);
      uint32_t at = uint32_t((pair * 0x9e3779b97f4a7c15ull) >> 52);
      while (key[at] != UINT64_MAX && key[at] != pair) at = (at + 1) % kPlaces;
      if (last[at] == from[k]) continue;  // the same point again
      last[at] = from[k];
      key[at] = pair;
      agreed += met[at]++;
      sampled++;
    }
    blocks = double(sampled) * double(sampled) / double(std::max<uint64_t>(agreed, 1)) + C;
    if (agreed >= 16 && 288 * blocks < kFarSystem / 2) break;
  }
  return blocks;
}

// The tracks of a problem, as prefer_schur weighs them.
Tracks survey(uint32_t C, uint32_t P, uint32_t M, const uint32_t* index) {
  Tracks t = count_pairs(index + 2 * size_t(M), P);
  if (288.0 * double(schur_block_bound(C, t.pairs)) > kFarSystem)
    t.spread = std::min(spread_blocks(C, P, M, index), double(schur_block_bound(C, t.pairs)));
  return t;
}

// The PCG steps of a solve to `tolerance` that the choice below counts on, from few: spheres, arcs and rings of
// 16 to 60 cameras took 8 to 19 steps at 1e-2, 10 to 30 at 1e-3 and 21 to 44 at 1e-6, 200 cameras 22, 36 and 68,
// 1,500 cameras 60, 66 and 75.
double expected_steps(uint64_t C, double tolerance) {
  return (10 + 8 * std::log10(1e-2 / tolerance)) * std::max(1.0, std::sqrt(double(C) / 60));
}

// Whether a solve forms the reduced system explicitly: its values cost about 0.04 ns a pair of observations of
// one point, once per linear solve, and a PCG step then a pass over the blocks (a sixth of their bound where
// cameras share points with their neighbours, at 8 TB/s from the L2) and two exchanges, against a pass over
// every observation (0.033 ns each) and five launches in a graph loop; compared over `most` PCG steps (16 for an
// LM iteration, 64 for the adjoint's tighter solves).  Six iterations on the product and on the system, ms:
// 331 cameras / 18,137 observations 7.7 and 2.8; 701 / 123,088 6.3 and 2.6; 1,301 / 61,318 8.5 and 5.2, /
// 369,365 8.0 and 5.1, / 1,106,971 12.7 and 7.1; 2,501 / 246,549 7.8 and 6.2, / 1,230,585 18.8 and 10.0; every
// camera seeing every point: 120 / 180,000 4.3 and 3.8, 200 / 600,000 6.0 and 14.1.
//
// A solve that its budget (of which it takes some 0.85) or its tolerance ends after few steps has less to gain.
// There a pair costs 0.036 ns where the records of a camera's neighbours (about eight times the pairs an
// observation has) lie in the 126 MB L2 together, else 0.046.  Six iterations again: 26 cameras / 2.1M
// observations of 12.5 pairs: budget 12 8.4 and 10.5, 16 10.1 and 10.7, 24 14.2 and 11.4; tolerance 1e-2 8.3 and
// 11.0.  200 cameras / 10M of 12.2 pairs: budget 16 41.8 and 52.8, 24 53.8 and 53.0.  600 cameras / 1.3M of 10.3:
// budget 8 5.3 and 5.6, 12 6.9 and 5.8.
//
// The system is FP64, so a mixed request is also weighed against its own product: 0.022 ns an observation where
// the first PCG run reaches the tolerance; where the budget ends the runs, their restarts make it 0.036 for each
// step of the budget.  The 26 cameras: tolerance 1e-2 7.8 and 11.0, 1e-3 9.4 and 11.1, 1e-6 16.9 and 11.3, budget
// 16 17.0 and 10.7; the 200 cameras: 1e-2 43.3 and 55.5, 2e-3 58.7 and 55.9.
//
// A track of n cameras makes n^2 blocks of S (each some 0.5 ns to write), which cost a step 0.04 ns each from
// shared memory or the L2 and 0.1 beyond; on the product its warp takes 0.04 us an observation.  Six iterations,
// every camera seeing every point: 300 cameras / 50 points 5.8 and 4.0, 400 / 30 6.4 and 4.0, 540 / 40 7.1 and 6.4,
// 600 / 30 8.0 and 11.5, 600 / 10 7.6 and 9.9.  (The adjoint's product is slower on these: 600 / 30 6.4 and 4.9 a
// call; it does not count them.)  Where any camera meets any other S is as large without long tracks: 600 cameras
// / 100,000 observations of 5 random cameras a point 6.2 and 5.7, 800 / 120,000 7.0 and 12.5, 1,500 / 1.0M 14.8 and
// 40.3; four iterations on 4,600 / 1.5M 17.4 and 90.7.
bool prefer_schur(uint64_t C, uint64_t M, Tracks tracks, uint32_t budget, double most, double expected, bool mixed) {
  const uint64_t pairs = tracks.pairs;
  if (6 * C + 1 > tba::product_max_unknowns() || pairs >= 0x7fffffffull || M > 0x0fffffffull) return false;
  const double seen = double(std::min<uint64_t>(tracks.longest, C)), spread = 288 * tracks.spread > kFarSystem ? tracks.spread : 0,
               dense = std::max(seen * seen, spread), bytes = 288 * dense;
  const double walk = std::max(288e-6 / 8 * double(schur_block_bound(C, pairs)) / 6,
                               (bytes < 90e6 ? 4e-5 : 1e-4) * dense);
  // A step's cost on the product less that on the system, at `k` us an observation.
  const auto step = [&](double k) { return 16 + std::max(k * double(M), 0.04 * tracks.longest) - walk; };
  const double write = 5e-4 * dense;
  if (!(4e-5 * double(pairs) + write < most * step(3.3e-5))) return false;
  const double reach = 144 * double(M) * std::min(1.0, 8 * double(pairs) / double(M) / double(C));
  const double form = (reach < 126e6 ? 3.6e-5 : 4.6e-5) * double(pairs) + write;
  if (mixed) return form < std::min(budget * step(3.6e-5), expected * step(2.2e-5));
  return form < std::min(0.85 * budget, expected) * step(3.3e-5);
}

// Device memory of a solve's explicit system beside the workspace: structure, segment sums, blocks.
// `blocks` and `camera_pairs` bound the blocks of S and the camera pairs.
struct SchurLayout {
  Layout L;
  size_t counts, bits, row_blk, row_pair, row_ptr, col, pairs, begin, rc, dst, seg_block, totals, part, S;
  size_t share, uni, uni_n, local, pbuf, zx, slots;  // the persistent PCG's
  uint32_t C, nchunks, seg = 0, grid = 1;
  uint64_t npairs, camera_pairs;
  // `all_pairs`: the pairs of all systems formed at once (0: this one alone), which size the segments.  (512
  // windows sized one by one, at 32 pairs a segment: 0.29 ms adding the ends and 1.40 ms the sums; sized
  // together: 0.05 and 1.48.)
  SchurLayout(uint32_t C, uint64_t npairs, uint32_t nchunks, int sms, uint64_t all_pairs = 0)
      : C(C), nchunks(nchunks), npairs(npairs), camera_pairs(std::min<uint64_t>(npairs, uint64_t(C) * (C + 1) / 2)) {
    const uint64_t blocks = schur_block_bound(C, npairs);
    // Pairs per warp of the block sums: a few warps' worth of segments on every SM.
    seg = tba::kPairSegMin;
    while (seg < tba::kPairSegMax && std::max(npairs, all_pairs) / seg > uint64_t(64) * uint64_t(sms)) seg *= 2;
    const size_t segs = size_t((npairs + seg - 1) / seg);
    const size_t bwords = (C + 31) / 32;
    counts = L.take<uint32_t>(size_t(nchunks) * C);
    bits = L.take<uint32_t>(C * bwords);
    row_blk = L.take<uint32_t>(C + 1);
    row_pair = L.take<uint32_t>(C + 1);
    row_ptr = L.take<uint32_t>(C + 1);
    col = L.take<uint32_t>(blocks);
    pairs = L.take<uint2>(npairs);
    begin = L.take<uint32_t>(camera_pairs + 1);
    rc = L.take<uint2>(camera_pairs);
    dst = L.take<uint2>(camera_pairs);
    seg_block = L.take<uint32_t>(segs);
    totals = L.take<uint32_t>(4);
    grid = tba::pcg_grid(blocks, C, sms);
    share = L.take<uint32_t>(grid + 1);
    uni = L.take<uint32_t>(size_t(grid) * C);
    uni_n = L.take<uint32_t>(grid);
    local = L.take<uint32_t>(blocks);
    pbuf = L.take<double>(size_t(grid) * 12 * C);
    zx = L.take<tba::Flagged>(6 * size_t(C));
    slots = L.take<tba::Flagged>(4 * size_t(grid));
    part = L.take<double>(72 * segs);
    S = L.take<double>(36 * blocks);
  }
  // The parts of the structure's and the PCG's parameters that lie in this memory.
  void bind(char* base, tba::SchurParams& q, tba::PcgSystem& a) const {
    auto u32 = [&](size_t off) { return reinterpret_cast<uint32_t*>(base + off); };
    auto u2 = [&](size_t off) { return reinterpret_cast<uint2*>(base + off); };
    auto f64 = [&](size_t off) { return reinterpret_cast<double*>(base + off); };
    q.C = a.C = C;
    q.nchunks = nchunks;
    q.bwords = (C + 31) / 32;
    q.seg = seg;
    q.max_pairs = uint32_t(npairs);
    q.max_blocks = uint32_t(camera_pairs);
    q.counts = u32(counts);
    q.bits = u32(bits);
    q.row_blk = u32(row_blk);
    q.row_pair = u32(row_pair);
    q.row_ptr = u32(row_ptr);
    q.col = u32(col);
    q.pairs = u2(pairs);
    q.blk_begin = u32(begin);
    q.blk_rc = u2(rc);
    q.blk_dst = u2(dst);
    q.seg_block = u32(seg_block);
    q.totals = u32(totals);
    q.part = f64(part);
    q.S = f64(S);
    a.S = q.S;
    a.max_blocks = uint32_t(std::min<uint64_t>(schur_block_bound(C, npairs), UINT32_MAX));
    a.row_ptr = q.row_ptr;
    a.col = q.col;
    a.share = u32(share);
    a.uni = u32(uni);
    a.uni_n = u32(uni_n);
    a.local = u32(local);
    a.pbuf = f64(pbuf);
    a.zx = reinterpret_cast<tba::Flagged*>(base + zx);
    a.slots = reinterpret_cast<tba::Flagged*>(base + slots);
  }
};

constexpr size_t kAllocationGrain = size_t(2) << 20;  // an allocation takes whole pages of the device's memory

// The device's free memory, with the explicit system's buffer given back when `need` takes it.
size_t free_memory(tba_device* d, size_t need) {
  size_t free_bytes = 0, total_bytes = 0;
  CUDA_TRY(cudaMemGetInfo(&free_bytes, &total_bytes));
  if (need > free_bytes && d->schur) {
    CUDA_TRY(cudaFree(d->schur));
    d->schur = nullptr;
    d->schur_capacity = 0;
    CUDA_TRY(cudaMemGetInfo(&free_bytes, &total_bytes));
  }
  return free_bytes;
}

// Whether the workspace and an explicit system's memory of these sizes fit the device, with what the
// handle holds given back where it has to grow.
bool memory_for(tba_device* d, size_t workspace, size_t schur) {
  if (d->capacity >= workspace && d->schur_capacity >= schur) return true;
  size_t free_bytes = 0, total_bytes = 0;
  CUDA_TRY(cudaMemGetInfo(&free_bytes, &total_bytes));
  const size_t held = (d->capacity < workspace ? d->capacity : 0) + (d->schur_capacity < schur ? d->schur_capacity : 0);
  const size_t need = (d->capacity < workspace ? workspace : 0) + (d->schur_capacity < schur ? schur : 0);
  return need <= free_bytes + held;
}

// Grows a device buffer kept by the handle to `bytes` (its old contents are dropped).
void grow(char*& buffer, size_t& capacity, size_t bytes, const char* what) {
  if (capacity >= bytes) return;
  if (buffer) CUDA_TRY(cudaFree(buffer));
  buffer = nullptr;
  capacity = 0;
  size_t free_bytes = 0, total_bytes = 0;
  CUDA_TRY(cudaMemGetInfo(&free_bytes, &total_bytes));
  if (bytes > free_bytes)
    throw Fail{TBA_ERROR_BUDGET, std::string(what) + " needs " + std::to_string(bytes) +
                                     " bytes of device memory, more than the working budget of " +
                                     std::to_string(free_bytes) + " bytes"};
  CUDA_TRY(cudaMalloc(&buffer, bytes));
  capacity = bytes;
}

// The handle's buffers for a call that needs these sizes.  A workspace that has to grow may need the
// memory of an explicit system that this call does not use.
void make_room(tba_device* d, size_t workspace, size_t schur, const char* what) {
  const bool both = d->capacity < workspace && d->schur_capacity < schur;
  if (d->schur && (both || (d->capacity < workspace && schur == 0))) {
    CUDA_TRY(cudaFree(d->schur));
    d->schur = nullptr;
    d->schur_capacity = 0;
  }
  grow(d->arena, d->capacity, workspace, what);
  grow(d->schur, d->schur_capacity, schur, what);
}

// Makes `loop` a graph of one while node whose body `capture(handle, stream)` records (returning its
// kernel count): kept when it was built for the same `key` (the launch parameters its kernels bake),
// built again otherwise.
template <class Capture>
cudaError_t build_device_loop(PcgLoop& loop, const void* key, size_t key_len, cudaStream_t s, Capture capture) {
  const char* bytes = static_cast<const char*>(key);
  if (loop.exec && loop.key.size() == key_len && std::memcmp(loop.key.data(), bytes, key_len) == 0)
    return cudaSuccess;
  loop.release();
  cudaError_t e = cudaGraphCreate(&loop.graph, 0);
  if (e != cudaSuccess) return e;
  // The condition starts at 1 at every launch: the body runs at least once (its kernels are no-ops
  // when the PCG is already stopped), then the body's last kernel decides.
  cudaGraphConditionalHandle handle;
  e = cudaGraphConditionalHandleCreate(&handle, loop.graph, 1, cudaGraphCondAssignDefault);
  if (e != cudaSuccess) return e;
  cudaGraphNodeParams np{};
  np.type = cudaGraphNodeTypeConditional;
  np.conditional.handle = handle;
  np.conditional.type = cudaGraphCondTypeWhile;
  np.conditional.size = 1;
  cudaGraphNode_t node;
  e = cudaGraphAddNode(&node, loop.graph, nullptr, 0, &np);
  if (e != cudaSuccess) return e;
  e = cudaStreamBeginCaptureToGraph(s, np.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                    cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return e;
  loop.body_kernels = capture(handle, s);
  const cudaError_t launched = cudaGetLastError();
  cudaGraph_t captured = nullptr;
  e = cudaStreamEndCapture(s, &captured);
  if (launched != cudaSuccess) return launched;
  if (e != cudaSuccess) return e;
  e = cudaGraphInstantiate(&loop.exec, loop.graph, 0);
  if (e != cudaSuccess) {
    loop.exec = nullptr;
    return e;
  }
  loop.key.assign(bytes, bytes + key_len);
  return cudaSuccess;
}

// The grid engine's PCG loop for the launch parameters `q`.
cudaError_t build_pcg_loop(PcgLoop& loop, const tba::Params& q, cudaStream_t s) {
  return build_device_loop(loop, &q, sizeof q, s, [&](cudaGraphConditionalHandle handle, cudaStream_t cs) {
    tba::Params body = q;
    body.pcg_loop = handle;
    tba::launch_product(body, cs);
    tba::launch_product_finish(body, cs);
    tba::launch_pcg_loop_next(body, cs);
    return uint32_t(q.factored ? 4 : 5) + 1;
  });
}

// The adjoint's PCG loop: the step kernels read neither the damping nor the right-hand side's mode,
// so one graph serves every linear solve of a vjp (and of the next call with the same arrays).
cudaError_t build_adjoint_loop(PcgLoop& loop, const tba::AdjParams& a, cudaStream_t s) {
  tba::AdjParams key = a;
  key.mu = 0;
  key.rhs_mode = 0;
  key.loop = 0;
  return build_device_loop(loop, &key, sizeof key, s, [&](cudaGraphConditionalHandle handle, cudaStream_t cs) {
    tba::AdjParams body = key;
    body.loop = handle;
    const uint32_t step = tba::adj_launch_pcg_step(body, cs);
    return step + tba::adj_launch_loop_next(body, cs);
  });
}

// Whether a device-side loop was built.  A driver that cannot build conditional graph nodes makes
// the handle run every later PCG from the host (the same kernels, launched in chunks); any other
// failure is the call's error.
bool device_loop_ready(tba_device* d, PcgLoop& loop, cudaError_t built) {
  if (built == cudaSuccess) return true;
  loop.release();
  if (built == cudaErrorNotSupported || built == cudaErrorStreamCaptureUnsupported) {
    cudaGetLastError();
    d->host_pcg_only = true;
    return false;
  }
  throw Fail{TBA_ERROR_CUDA, std::string("device PCG loop: ") + cudaGetErrorString(built)};
}

cudaEvent_t event(tba_device* d, size_t k) {
  while (d->events.size() <= k) {
    cudaEvent_t e;
    CUDA_TRY(cudaEventCreate(&e));
    d->events.push_back(e);
  }
  return d->events[k];
}

// The host-side schedules of one problem's index: warp tasks (with their first observations),
// camera chunks and the number of fixed cameras.
struct HostPlan {
  std::vector<uint32_t> tasks, task_obs;
  Chunks chunks;
  uint32_t fixed = 0;
  Tracks tracks;  // a resident scene's
  // The arrays a solve uploads, in the order of a resident scene's device copy.
  std::vector<const std::vector<uint32_t>*> sections() const {
    return {&tasks, &task_obs, &chunks.cam, &chunks.beg, &chunks.cam_first};
  }
};

HostPlan make_plan(const tba_control* ctl, const uint32_t* index, int sms) {
  const uint32_t C = ctl->cameras, P = ctl->points, M = ctl->observations;
  const uint32_t* ps = index + 2 * size_t(M);
  const uint32_t* cs = ps + P + 1;
  const uint32_t* active = cs + C + 1 + M;
  HostPlan plan;
  plan.tasks = build_tasks(ps, P);
  plan.task_obs.resize(plan.tasks.size());
  for (size_t t = 0; t < plan.tasks.size(); t++) plan.task_obs[t] = ps[plan.tasks[t]];
  plan.chunks = build_chunks(cs, C, chunk_size(M, sms));
  for (uint32_t c = 0; c < C; c++) plan.fixed += active[c] == 0;
  return plan;
}

// Blocks of the acceptance: each adds the task blocks' costs again, so there are few of them, each with
// a few thousand values of the candidate to copy.
uint32_t commit_grid(uint32_t C, uint32_t P) {
  return uint32_t(std::min<uint64_t>(592, std::max<uint64_t>(1, (std::max<uint64_t>(12ull * C, 3ull * P) + 2047) / 2048)));
}

// The explicit system's structure, values and PCG of one problem, from the problem's parameters; the
// problem takes the system's blocks.
void bind_problem(tba::Params& p, tba::SchurParams& q, tba::PcgSystem& a) {
  q.M = p.M;
  q.obs_camera = p.obs_camera;
  q.obs_point = p.obs_point;
  q.point_start = p.point_start;
  q.camera_obs = p.camera_obs;
  q.active = p.active;
  q.chunk_cam = p.chunk_cam;
  q.chunk_beg = p.chunk_beg;
  q.cam_chunk = p.cam_chunk;
  q.A = p.A;
  q.go = p.state + tba::S_ACTIVE;
  p.S = q.S;
  p.row_ptr = q.row_ptr;
  p.col = q.col;
  a.shared = p.shared;
  a.Minv = p.camMinv;
  a.scf = p.camScf;
  a.x = p.x;
  a.r = p.r;
  a.z = p.z;
  a.p = p.p;
  a.state = p.state;
  a.active = tba::S_CG_ACTIVE;
  a.failed = tba::S_CG_FAILED;
  a.converged = tba::S_CG_CONVERGED;
  a.rho = tba::S_RHO;
  a.r0 = tba::S_R0;
  a.r2 = tba::S_R2;
  a.inner_r0 = tba::S_INNER_R0;
  a.steps = tba::S_CG_SOLVE_STEPS;
  a.all_steps = tba::S_CG_STEPS;
  a.wait = tba::S_WAIT;
  a.focal_diag = tba::S_FOCAL_SFF;
  a.focal_inv = tba::S_FOCAL_INV;
  a.tol = p.tol;
  a.tol_inner = p.tol_inner;
  a.alpha_limit = 1e20;
  a.rhs = p.camRhs;
  a.scal_part = p.scal_part;
  a.scal_blocks = p.task_blocks;
  a.solving = tba::S_ACTIVE;
  a.block_failed = tba::S_POINT_FAILED;
  a.lambda = tba::S_LAMBDA;
  a.focal_full = tba::S_FOCAL_DIAG;
  a.focal_rhs = tba::S_FOCAL_RHS;
  a.clear_from = tba::S_RHO;
  a.clear_to = 25;
}

// Where a solve reads its problem and where it leaves the solution.  With `device_source` the
// scene and index are device pointers (a resident scene) and `plan` is given; `writeback` (device)
// receives the solved poses and points; `output` may be null and `state` (host) receives the
// result's state words.
struct SolveIO {
  bool device_source = false;
  const HostPlan* plan = nullptr;
  double* writeback = nullptr;
  double* state = nullptr;
  // When set, the O(M) checks run on the device right after the upload and a failure is raised
  // (with these host-side results, in the serial order) before any solver kernel runs.
  const HostChecks* checks = nullptr;
  double* check_ms = nullptr;  // receives the device checks' host wall time
  // With `plan`: a device copy of its arrays (HostPlan::sections, concatenated), copied on the
  // device instead of uploaded.
  const uint32_t* plan_dev = nullptr;
};

void solve(tba_device* d, const tba_control* ctl, const double* scene, const uint32_t* index,
           double* output, tba_report* report, const SolveIO& io = SolveIO()) {
  const auto wall0 = std::chrono::steady_clock::now();
  const uint32_t C = ctl->cameras, P = ctl->points, M = ctl->observations;
  const bool shared = ctl->shared_focal != 0;
  const uint32_t m = 6 * C + (shared ? 1 : 0);
  // The host schedules (warp tasks, camera chunks) are built while the problem arrays upload: the
  // workspace is laid out with bounds of their sizes (at most P + 1 task starts; at most
  // C + M / 128 + 1 chunks, chunks being at least 128 observations long).  A problem whose camera
  // offsets fail the host checks gets no schedule; its checks fail before any kernel runs.
  const bool plannable = !io.checks || (!io.checks->camera_ends && !io.checks->camera_offsets);
  const uint64_t max_tasks = io.plan ? io.plan->tasks.size() : uint64_t(P) + 1;
  const uint64_t max_chunks = io.plan ? io.plan->chunks.cam.size() : uint64_t(C) + M / 128 + 1;

  Params p{};
  p.C = C;
  p.P = P;
  p.M = M;
  p.D = ctl->directional_points;
  p.m = m;
  p.anchor = ctl->anchor;
  p.scale_view = ctl->scale_view;
  p.shared = shared;
  p.huber = ctl->huber;
  p.tol = ctl->cg_tolerance;
  p.stall = ctl->stall_tolerance;
  const uint32_t max_task_blocks = std::max<uint32_t>(1, 4 * uint32_t(d->sms));
  const uint32_t fblocks = tba::product_finish_blocks(p);
  // The one-pass product over stored factors when its camera sums fit shared memory; the two-pass
  // recompute form otherwise.  The mixed form stores FP32 factors for its PCG and FP64 factors for
  // its refinement residual, its FP64 tail and the back-substitution.
  p.factored = m <= tba::product_max_unknowns();
  p.Mpad = (M + 31) / 32 * 32;
  // The explicit reduced system takes the place of the product over stored factors where it costs less than
  // the product of the form asked for and fits the device; it is FP64, so a mixed request then needs no refinement.
  // (Without iterations there is no system to form: its structure alone took 0.03 ms at 7 cameras and 0.35 at
  // 1,500 and 1.8M observations, of calls of 0.21 and 5.9 ms.)
  const Tracks tracks = ctl->iterations == 0 ? Tracks() : (io.plan ? io.plan->tracks : survey(C, P, M, index));
  const uint64_t npairs = tracks.pairs;
  // (The product's error asked of a mixed request is the FP32 product's.)
  const bool keep_product = ctl->precision == TBA_PRECISION_MIXED && (ctl->flags & TBA_FLAG_PRODUCT_ERROR) != 0;
  bool schur = p.factored && ctl->iterations > 0 && !keep_product &&
               prefer_schur(C, M, tracks, ctl->max_cg, 16, expected_steps(C, ctl->cg_tolerance),
                            ctl->precision == TBA_PRECISION_MIXED);
  bool mixed = false;
  size_t factor_bytes = 0, factor32_bytes = 0;
  uint32_t max_prod_blocks = 1;
  Layout L;
  size_t o_poses, o_points, o_cams, o_pixels, o_tposes, o_tpoints, o_index, o_pblk32, o_tasks, o_tobs, o_ccam, o_cbeg,
      o_cfirst, o_rlim, o_cmp, o_cmx, o_pblk, o_y, o_cprod, o_F, o_F32, o_pw, o_xw, o_acc, o_U, o_Minv, o_rhs, o_hcf,
      o_scf, o_chunk, o_vec, o_blk, o_scal, o_cost, o_ticket, o_state, o_out, o_keys, o_diag;
  auto lay_out = [&]() {
    mixed = ctl->precision == TBA_PRECISION_MIXED && !schur;
    factor_bytes = schur ? 18 * size_t(M) * 8 : (p.factored ? size_t(tba::kFactors) * p.Mpad * 8 : 0);
    factor32_bytes = p.factored && mixed ? size_t(tba::kFactors) * p.Mpad * 4 : 0;
    p.F = nullptr;
    p.F32 = mixed && p.factored ? reinterpret_cast<float*>(1) : nullptr;  // set below; selects the occupancy query
    const int per_sm = p.factored && !schur ? tba::product_blocks_per_sm(p) : 1;
    max_prod_blocks = schur ? 0 : std::max<uint32_t>(1, uint32_t(per_sm * d->sms));
    L = Layout();
    o_poses = L.take<double>(12 * size_t(C));
    o_points = L.take<double>(3 * size_t(P));
    o_cams = L.take<double>(6 * size_t(C));
    o_pixels = L.take<double>(2 * size_t(M));
    o_tposes = L.take<double>(12 * size_t(C));
    o_tpoints = L.take<double>(3 * size_t(P));
    o_index = L.take<uint32_t>(3 * size_t(M) + P + 2 * size_t(C) + 2);
    o_pblk32 = L.take<float>(mixed && p.factored ? 6 * size_t(P) : 0);
    o_tasks = L.take<uint32_t>(max_tasks);
    o_tobs = L.take<uint32_t>(max_tasks);
    o_ccam = L.take<uint32_t>(max_chunks);
    o_cbeg = L.take<uint32_t>(max_chunks + 1);
    o_cfirst = L.take<uint32_t>(C + 1);
    o_rlim = L.take<double>(C);
    o_cmp = L.take<uint32_t>(M);
    o_cmx = L.take<double>(2 * size_t(M));
    o_pblk = L.take<double>(12 * size_t(P));
    o_y = L.take<double>(4 * size_t(P));
    o_cprod = L.take<double>(8 * max_chunks);
    o_F = L.take<char>(factor_bytes);
    o_F32 = L.take<char>(factor32_bytes);
    o_pw = L.take<double>(6 * size_t(C));
    o_xw = L.take<double>(6 * size_t(C));
    o_acc = L.take<double>(p.factored ? size_t(max_prod_blocks) * m : 0);
    o_U = L.take<double>(21 * size_t(C));
    o_Minv = L.take<double>(36 * size_t(C));
    o_rhs = L.take<double>(6 * size_t(C));
    o_hcf = L.take<double>(6 * size_t(C));
    o_scf = L.take<double>(6 * size_t(C));
    o_chunk = L.take<double>(size_t(schur ? tba::kCameraPartialsExplicit : tba::kCameraPartials) * max_chunks);
    o_vec = L.take<double>(5 * size_t(m));
    o_blk = L.take<double>(4 * size_t(fblocks));
    o_scal = L.take<double>(size_t(tba::kScalarPartials) * max_task_blocks);
    o_cost = L.take<double>(4 * size_t(max_task_blocks));
    o_ticket = L.take<uint32_t>(8);
    o_state = L.take<double>(tba::S_WORDS);
    o_out = L.take<double>(12 * size_t(C) + 3 * size_t(P) + 27);
    o_keys = L.take<unsigned long long>(tba::CK_WORDS);
    o_diag = L.take<double>((ctl->flags & TBA_FLAG_PRODUCT_ERROR) ? 2 * size_t(m) : 0);
  };
  lay_out();
  if (schur) {
    // What the explicit system would add: when it does not fit, the product over stored factors.
    if (!memory_for(d, L.bytes, SchurLayout(C, npairs, uint32_t(max_chunks), d->sms).L.bytes)) {
      schur = false;
      lay_out();
    }
  }
  make_room(d, L.bytes, 0, "GPU BA");
  char* a = d->arena;
  auto D = [&](size_t off) { return reinterpret_cast<double*>(a + off); };
  auto U32 = [&](size_t off) { return reinterpret_cast<uint32_t*>(a + off); };
  p.poses = D(o_poses);
  p.points = D(o_points);
  p.cams = D(o_cams);
  p.pixels = D(o_pixels);
  p.tposes = D(o_tposes);
  p.tpoints = D(o_tpoints);
  uint32_t* dindex = U32(o_index);
  p.obs_camera = dindex;
  p.obs_point = dindex + M;
  p.point_start = dindex + 2 * size_t(M);
  p.camera_start = p.point_start + P + 1;
  p.camera_obs = p.camera_start + C + 1;
  p.active = p.camera_obs + M;
  p.pblk32 = mixed && p.factored ? reinterpret_cast<float*>(a + o_pblk32) : nullptr;
  p.tasks = U32(o_tasks);
  p.task_obs = U32(o_tobs);
  p.chunk_cam = U32(o_ccam);
  p.chunk_beg = U32(o_cbeg);
  p.cam_chunk = U32(o_cfirst);
  p.rlim = D(o_rlim);
  p.cm_point = U32(o_cmp);
  p.cm_pixel = D(o_cmx);
  p.pblk = D(o_pblk);
  p.y = D(o_y);
  p.chunk_prod = D(o_cprod);
  p.F = p.factored && !schur ? D(o_F) : nullptr;
  p.schur = schur;
  p.A = schur ? D(o_F) : nullptr;
  p.camScf = D(o_scf);
  p.F32 = p.factored && mixed ? reinterpret_cast<float*>(a + o_F32) : nullptr;
  p.pw = D(o_pw);
  p.xw = D(o_xw);
  p.acc_part = D(o_acc);
  p.camU = D(o_U);
  p.camMinv = D(o_Minv);
  p.camRhs = D(o_rhs);
  p.camHcf = D(o_hcf);
  p.chunk_part = D(o_chunk);
  double* vec = D(o_vec);
  p.x = vec;
  p.r = vec + m;
  p.p = vec + 2 * size_t(m);
  p.Sp = vec + 3 * size_t(m);
  p.z = vec + 4 * size_t(m);
  p.blk_part = D(o_blk);
  p.scal_part = D(o_scal);
  p.cost_part = D(o_cost);
  p.ticket = U32(o_ticket);
  p.state = D(o_state);
  p.output = D(o_out);

  // The mixed form's inner PCG runs stop at a relative residual the FP32 product can reach; the
  // FP64 refinement then measures the true residual against the caller's tolerance.
  p.tol_inner = mixed ? std::max(ctl->cg_tolerance, 1e-6) : ctl->cg_tolerance;

  cudaStream_t s = d->stream;
  size_t ev = 0;
  cudaEvent_t e_start = event(d, ev++), e_up = event(d, ev++), e_solved = event(d, ev++), e_down = event(d, ev++);
  uint64_t h2d = 0;
  // Problem arrays: host-to-device, or device-to-device from a resident scene.
  auto up = [&](void* dst, const void* src, size_t bytes) {
    if (bytes) CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, io.device_source ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, s));
    if (!io.device_source) h2d += bytes;
  };
  auto up_host = [&](void* dst, const void* src, size_t bytes) {
    if (bytes) CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
    h2d += bytes;
  };
  CUDA_TRY(cudaEventRecord(e_start, s));
  up(p.poses, scene, 12 * sizeof(double) * C);
  up(p.points, scene + 12 * size_t(C), 3 * sizeof(double) * P);
  up(const_cast<double*>(p.cams), scene + 12 * size_t(C) + 3 * size_t(P), 6 * sizeof(double) * C);
  up(const_cast<double*>(p.pixels), scene + 18 * size_t(C) + 3 * size_t(P), 2 * sizeof(double) * M);
  up(dindex, index, sizeof(uint32_t) * (3 * size_t(M) + P + 2 * size_t(C) + 2));
  // The schedules, built on the host while the copies above run.
  HostPlan own;
  if (!io.plan && plannable) own = make_plan(ctl, index, d->sms);
  const HostPlan& plan = io.plan ? *io.plan : own;
  const std::vector<uint32_t>& tasks = plan.tasks;
  const Chunks& chunks = plan.chunks;
  const uint32_t ntasks = tasks.empty() ? 0 : uint32_t(tasks.size() - 1), nchunks = uint32_t(chunks.cam.size());
  if (plannable) {
    if (tasks.size() > max_tasks || nchunks > max_chunks) throw Fail{TBA_ERROR_INTERNAL, "GPU BA schedule exceeds its bound"};
    // The plan's arrays: from the host, or from a resident scene's device copy.
    const size_t dst[5] = {o_tasks, o_tobs, o_ccam, o_cbeg, o_cfirst};
    size_t at = 0;
    const auto sections = plan.sections();
    for (size_t k = 0; k < sections.size(); k++) {
      const std::vector<uint32_t>& v = *sections[k];
      if (!v.empty()) {
        if (io.plan_dev)
          CUDA_TRY(cudaMemcpyAsync(U32(dst[k]), io.plan_dev + at, sizeof(uint32_t) * v.size(), cudaMemcpyDeviceToDevice, s));
        else
          up_host(U32(dst[k]), v.data(), sizeof(uint32_t) * v.size());
      }
      at += v.size();
    }
  }
  p.normalize_scale = plan.fixed == 1;
  p.ntasks = ntasks;
  p.nchunks = nchunks;
  p.task_blocks = std::max<uint32_t>(1, std::min<uint32_t>(max_task_blocks, (ntasks + 7) / 8));
  p.commit_blocks = commit_grid(C, P);
  p.prod_blocks = std::max<uint32_t>(1, std::min<uint32_t>(max_prod_blocks, (ntasks + 15) / 16));
  CUDA_TRY(cudaEventRecord(e_up, s));
  if (io.checks) {
    const auto c0 = std::chrono::steady_clock::now();
    // (claims: scratch until k_setup writes the camera-major point index)
    auto spent = [&] {
      if (io.check_ms)
        *io.check_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - c0).count();
    };
    try {
      device_checks(d, *io.checks, C, P, M, dindex, {p.poses, p.points, p.cams, p.pixels}, p.cm_point,
                    reinterpret_cast<unsigned long long*>(a + o_keys));
    } catch (...) {
      spent();
      throw;
    }
    spent();
    if (!plannable) throw Fail{TBA_ERROR_INTERNAL, "GPU BA checks passed a problem without a schedule"};
  }

  uint32_t launches = 0, lm_done = 0, refinements = 0, fp64_iterations = 0;
  tba::SchurParams sq{};
  tba::PcgSystem ps{};
  uint32_t pcg_blocks = 0;
  if (schur) {
    const SchurLayout Q(C, npairs, nchunks, d->sms);
    grow(d->schur, d->schur_capacity, Q.L.bytes, "GPU BA");
    Q.bind(d->schur, sq, ps);
    bind_problem(p, sq, ps);
    ps.polls = d->pcg_polls();
    launches += tba::schur_launch_structure(sq, s);
    pcg_blocks = Q.grid;
    launches += tba::pcg_launch_plan(ps, pcg_blocks, s);
    CUDA_TRY(cudaGetLastError());
  }
  // Mixed form: once an LM iteration's PCG needed the FP64 tail, the rest of the solve solves on the
  // FP64 product (the FP32 product does not reach the tolerance on such a system, and its restarts
  // would only add PCG runs).
  bool fp64_only = false;
  // Event pairs around the Schur products; after the solve, only the products that ran PCG steps
  // (the first `steps` of each LM iteration; later ones are guarded no-ops) count.
  std::vector<std::pair<size_t, size_t>> product_events;
  std::vector<std::pair<size_t, uint32_t>> product_spans;  // (first event pair, real steps) per LM iteration
  const bool time_products = (ctl->flags & TBA_FLAG_TIME_PRODUCTS) != 0;
  const bool diagnose = (ctl->flags & TBA_FLAG_PRODUCT_ERROR) != 0;
  const bool host_loop = time_products || (ctl->flags & TBA_FLAG_HOST_PCG_LOOP) != 0;
  // With the explicit system nothing in an iteration needs the host, so iterations are issued one ahead
  // of the last state read.
  const bool ahead = schur && !host_loop && !diagnose;
  // On the explicit system a mixed request's one run has the budgets of the mixed form's runs together, so that
  // a budget that the form's restarts make do with is enough here too (a run that it ends is a failed solve).
  constexpr uint32_t kFp32Restarts = 2;
  const uint32_t pcg_budget = ctl->max_cg * (schur && ctl->precision == TBA_PRECISION_MIXED ? kFp32Restarts + 2 : 1);
  cudaEvent_t read_done[2] = {event(d, ev), event(d, ev + 1)};
  ev += 2;
  // Kernels per step of the device-side PCG loop launched last, while its step count is unread.
  uint32_t loop_kernels = 0;
  tba::launch_initialize(p, s);
  tba::launch_cost(p, s);
  tba::launch_finish_metrics(p, s);
  launches += 4;
  CUDA_TRY(cudaGetLastError());
  bool lm_active = read_word(d, p.state, tba::S_ACTIVE) != 0;
  // The mixed form's FP64 tail: the one-pass product over the FP64 factors (the two-pass recompute
  // product when the engine keeps no factors).
  tba::Params tail = p;
  tail.F32 = nullptr;
  tail.tol_inner = 0;  // the tail stops at the solve's own tolerance
  double product_error_max = 0, product_error_norm = 0;
  for (uint32_t it = 0; it < ctl->iterations && lm_active; it++) {
    tba::launch_point_pass(p, s);
    tba::launch_camera_pass(p, s);
    tba::launch_camera_finish(p, s);
    if (schur) launches += tba::schur_launch_values(sq, s);
    launches += 3;
    if (!schur || host_loop || diagnose) {  // (the persistent PCG starts itself)
      tba::launch_pcg_init(p, s);
      launches++;
    }
    if (it == 0 && diagnose && read_word(d, p.state, tba::S_CG_ACTIVE) != 0) {
      // The solve's own product and the FP64 two-pass product on the first PCG direction.
      double* own = D(o_diag);
      double* ref = own + m;
      tba::Params fp64 = p;
      fp64.F32 = nullptr;
      fp64.factored = 0;
      tba::launch_product(p, s);
      if (schur) CUDA_TRY(cudaMemcpyAsync(own, p.Sp, m * sizeof(double), cudaMemcpyDeviceToDevice, s));
      else tba::launch_product_rows(p, own, s);
      tba::launch_product(fp64, s);
      tba::launch_product_rows(fp64, ref, s);
      launches += p.factored ? 5 : 6;
      CUDA_TRY(cudaGetLastError());
      std::vector<double> a(m), b(m);
      CUDA_TRY(cudaMemcpyAsync(a.data(), own, m * sizeof(double), cudaMemcpyDeviceToHost, s));
      CUDA_TRY(cudaMemcpyAsync(b.data(), ref, m * sizeof(double), cudaMemcpyDeviceToHost, s));
      CUDA_TRY(cudaStreamSynchronize(s));
      double dmax = 0, bmax = 0, d2 = 0, b2 = 0;
      for (uint32_t j = 0; j < m; j++) {
        const double e = a[j] - b[j];
        dmax = std::max(dmax, std::fabs(e));
        bmax = std::max(bmax, std::fabs(b[j]));
        d2 += e * e;
        b2 += b[j] * b[j];
      }
      product_error_max = bmax > 0 ? dmax / bmax : dmax;
      product_error_norm = b2 > 0 ? std::sqrt(d2 / b2) : std::sqrt(d2);
    }
    // PCG runs.  By default a run is one launch of the form's device-side PCG loop, which ends on the
    // device; its step count is taken from the next state read (every run is followed by one in the
    // same LM iteration).  With the host loop (timed products, or on request) the steps run in
    // chunks of guarded iterations, events around each product when timed; the read after each
    // chunk only ends the loop early.
    uint32_t done = 0, steps_before = 0;
    // `q` selects the product: the engine's own (FP32 factors in the mixed form), or the FP64
    // product of the mixed form's tail.  Only the engine's own products are timed.
    auto run_pcg = [&](uint32_t budget, const tba::Params& q, bool timed) {
      if (schur && !host_loop) {
        tba::PcgSystem a = ps;
        if (diagnose) a.rhs = nullptr;  // k_pcg_init has run
        CUDA_TRY(tba::launch_pcg(a, budget, pcg_blocks, s));
        launches++;
        return;
      }
      if (!host_loop && !d->host_pcg_only) {
        if (budget <= done) return;
        PcgLoop& loop = d->pcg_loops[&q == &p ? 0 : 1];
        if (device_loop_ready(d, loop, build_pcg_loop(loop, q, s))) {
          tba::launch_pcg_loop_begin(q, budget - done, s);
          launches++;
          CUDA_TRY(cudaGraphLaunch(loop.exec, s));
          loop_kernels = loop.body_kernels;
          return;
        }
      }
      const size_t first_pair = product_events.size();
      uint32_t chunk = 8;
      while (done < budget) {
        const uint32_t k = std::min(chunk, budget - done);
        for (uint32_t j = 0; j < k; j++) {
          if (time_products && timed) {
            const size_t e0 = ev++, e1 = ev++;
            CUDA_TRY(cudaEventRecord(event(d, e0), s));
            tba::launch_product(q, s);
            CUDA_TRY(cudaEventRecord(event(d, e1), s));
            product_events.emplace_back(e0, e1);
          } else {
            tba::launch_product(q, s);
          }
          tba::launch_product_finish(q, s);
          launches += schur ? 3 : (q.factored ? 4 : 5);
        }
        CUDA_TRY(cudaGetLastError());
        done += k;
        if (done >= budget || read_word(d, p.state, tba::S_CG_ACTIVE) == 0) break;
        chunk = std::min<uint32_t>(2 * chunk, 32);
      }
      // The products of this run that did PCG steps (later launches of a chunk are no-ops).
      const uint32_t steps = uint32_t(read_word(d, p.state, tba::S_CG_SOLVE_STEPS));
      if (time_products && timed) product_spans.emplace_back(first_pair, steps - steps_before);
      steps_before = steps;
    };
    // After a state read: the steps of the device-side PCG loop that ran before it.
    auto account_loop = [&]() {
      if (!loop_kernels) return;
      const uint32_t iters = uint32_t(d->pinned[tba::S_LOOP_ITERS]);
      done += iters;
      launches += iters * loop_kernels;
      loop_kernels = 0;
    };
    if (fp64_only) fp64_iterations++;
    run_pcg(pcg_budget, fp64_only ? tail : p, !fp64_only);
    // Mixed form: FP64 iterative refinement.  The true (FP64) residual of the FP32-product solution
    // restarts the PCG from that solution when it is above the tolerance; a restarted run (with an
    // iteration budget of its own) uses the FP32 product again and is checked again.  Only a
    // solution still above the tolerance after kFp32Restarts such runs is finished on the FP64
    // product, which resolves what FP32 factors cannot on badly conditioned systems.
    if (mixed && !fp64_only) {
      for (uint32_t round = 0;; round++) {
        tba::launch_refine(p, s);
        launches += 4;
        CUDA_TRY(cudaGetLastError());
        const bool active = read_word(d, p.state, tba::S_CG_ACTIVE) != 0;
        account_loop();
        if (!active) break;
        refinements++;
        if (round < kFp32Restarts) {
          run_pcg(done + ctl->max_cg, p, true);
          continue;
        }
        run_pcg(done + ctl->max_cg, tail, false);
        fp64_only = true;
        break;
      }
    }
    tba::launch_update_cameras(p, s);
    tba::launch_update_points(p, s);
    tba::launch_accept(p, s);
    launches += 3;
    CUDA_TRY(cudaGetLastError());
    lm_done++;
    if (ahead) {
      // The state goes to the host while the next iteration, a no-op should this one have ended the solve,
      // is issued.
      double* words = d->pinned + tba::S_READ * (it & 1);
      CUDA_TRY(cudaMemcpyAsync(words, p.state, tba::S_READ * sizeof(double), cudaMemcpyDeviceToHost, s));
      CUDA_TRY(cudaEventRecord(read_done[it & 1], s));
      if (it > 0) {
        CUDA_TRY(cudaEventSynchronize(read_done[(it - 1) & 1]));
        check_waits(d->pinned + tba::S_READ * ((it - 1) & 1));
        lm_active = d->pinned[tba::S_READ * ((it - 1) & 1) + tba::S_ACTIVE] != 0;
      }
      continue;
    }
    lm_active = read_word(d, p.state, tba::S_ACTIVE) != 0;
    account_loop();
  }
  if (ahead) {
    // Iterations that ran: the accepted and rejected steps.
    if (read_word(d, p.state, tba::S_ACCEPTED) >= 0)
      lm_done = uint32_t(d->pinned[tba::S_ACCEPTED] + d->pinned[tba::S_REJECTED]);
  }
  tba::launch_pack(p, s);
  launches++;
  CUDA_TRY(cudaGetLastError());
  CUDA_TRY(cudaEventRecord(e_solved, s));
  const size_t out_len = 12 * size_t(C) + 3 * size_t(P) + 26 + (shared ? 1 : 0);
  const size_t state_len = 26 + (shared ? 1 : 0);
  size_t d2h = 0;
  if (output) {
    CUDA_TRY(cudaMemcpyAsync(output, p.output, out_len * sizeof(double), cudaMemcpyDeviceToHost, s));
    d2h += out_len * sizeof(double);
  }
  if (io.state) {
    CUDA_TRY(cudaMemcpyAsync(io.state, p.output + 12 * size_t(C) + 3 * size_t(P), state_len * sizeof(double),
                             cudaMemcpyDeviceToHost, s));
    d2h += state_len * sizeof(double);
  }
  if (io.writeback) {
    CUDA_TRY(cudaMemcpyAsync(io.writeback, p.poses, 12 * sizeof(double) * C, cudaMemcpyDeviceToDevice, s));
    CUDA_TRY(cudaMemcpyAsync(io.writeback + 12 * size_t(C), p.points, 3 * sizeof(double) * P, cudaMemcpyDeviceToDevice, s));
  }
  CUDA_TRY(cudaEventRecord(e_down, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  if (report) {
    std::memset(report, 0, sizeof *report);
    float ms = 0;
    CUDA_TRY(cudaEventElapsedTime(&ms, e_start, e_up));
    report->upload_ms = ms;
    CUDA_TRY(cudaEventElapsedTime(&ms, e_up, e_solved));
    report->solve_ms = ms;
    CUDA_TRY(cudaEventElapsedTime(&ms, e_solved, e_down));
    report->download_ms = ms;
    double total = 0;
    uint32_t counted = 0;
    for (size_t k = 0; k < product_spans.size(); k++) {
      const size_t end = k + 1 < product_spans.size() ? product_spans[k + 1].first : product_events.size();
      const size_t last = std::min(end, product_spans[k].first + product_spans[k].second);
      for (size_t j = product_spans[k].first; j < last; j++) {
        CUDA_TRY(cudaEventElapsedTime(&ms, d->events[product_events[j].first], d->events[product_events[j].second]));
        total += ms;
        counted++;
      }
    }
    report->product_ms = total;
    report->product_launches = counted;
    report->h2d_bytes = h2d;
    report->d2h_bytes = d2h;
    report->kernel_launches = launches;
    report->lm_iterations = lm_done;
    const double* st = output ? output + 12 * size_t(C) + 3 * size_t(P) : io.state;
    report->cg_iterations = st ? uint32_t(st[tba::S_CG_STEPS]) : 0;
    report->engine = schur ? 2 : (p.factored ? 0 : 1);
    report->product_blocks = p.factored && !schur ? p.prod_blocks : 0;
    report->refinements = uint32_t(refinements);
    report->fp64_iterations = fp64_iterations;
    report->product_error_max = product_error_max;
    report->product_error_norm = product_error_norm;
    report->wall_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - wall0).count();
  }
}

// ---- batched local-window solves ------------------------------------------------------------------

// The caller's arrays of one batched problem, checked as tba_bundle_adjust checks a problem.
tba_control batch_problem_control(const tba_batch_control* bc, const tba_batch_problem& q) {
  tba_control c{};
  c.cameras = q.cameras;
  c.points = q.points;
  c.directional_points = 0;
  c.observations = q.observations;
  c.anchor = q.anchor;
  c.scale_view = q.scale_view;
  c.iterations = bc->iterations;
  c.max_cg = bc->max_cg;
  c.shared_focal = bc->shared_focal;
  c.precision = bc->precision;
  c.flags = 0;
  c.huber = bc->huber;
  c.cg_tolerance = bc->cg_tolerance;
  c.stall_tolerance = bc->stall_tolerance;
  return c;
}

// One problem of a batch as the host schedules it.
struct WindowPlan {
  std::vector<uint32_t> tasks;
  Chunks chunks;
  uint64_t pairs = 0;
};

struct BatchReport {
  int shape = 0;
  uint32_t threads = 0, blocks = 0, launches = 0;
  bool replayed = false, mixed = false;
};

// The batch on the grid kernels: every kernel of an LM iteration runs over all problems at once (its
// blocks a list of (problem, block)), with each problem's reduced system explicit and its PCG in one
// block; the iteration is a CUDA graph, replayed while the batch's lists keep their places.  With
// `whole_check` the device checks the arrays first, and the host's checks give the message.  False
// (nothing launched) when the workspace does not fit.
bool batch_on_grid(tba_device* d, const tba_batch_control* bc, const tba_batch_problem* probs, uint32_t count,
                   const std::vector<WindowPlan>& plans, const std::vector<uint32_t>& order, const double* scene,
                   size_t scene_len, const uint32_t* index, size_t index_len, size_t output_len, cudaEvent_t uploaded,
                   cudaEvent_t begun, BatchReport& rep, double*& dout_of, uint64_t& h2d,
                   const std::function<void()>* whole_check) {
  const bool shared = bc->shared_focal != 0;
  Layout L;
  const size_t o_scene = L.take<double>(scene_len), o_index = L.take<uint32_t>(index_len), o_out = L.take<double>(output_len);
  // The plans' arrays, then the lists of blocks, in one upload.
  std::vector<uint32_t> flat;
  struct Place {
    size_t tasks, obs, cam, beg, first;
  };
  std::vector<Place> places(count);
  uint64_t tasks_total = 0;
  for (uint32_t k = 0; k < count; k++) tasks_total += plans[k].tasks.size() - 1;
  // Tasks per warp of the task kernels: a few waves of blocks over the batch, up to eight.
  const uint32_t per_warp = uint32_t(std::min<uint64_t>(8, std::max<uint64_t>(1, tasks_total / (8 * 8 * uint64_t(d->sms)))));
  std::vector<uint2> lists[10];  // one, task, chunk, finish, setup, commit, pack | camera, pairs, sums
  std::vector<SchurLayout> systems;
  systems.reserve(count);
  uint32_t Cmax = 2;
  uint64_t all_pairs = 0;
  for (uint32_t k = 0; k < count; k++) all_pairs += plans[k].pairs;
  for (uint32_t k = 0; k < count; k++) {
    const tba_batch_problem& q = probs[k];
    const WindowPlan& w = plans[k];
    Place& at = places[k];
    const uint32_t* ps = index + q.index_offset + 2 * size_t(q.observations);
    at.tasks = flat.size();
    flat.insert(flat.end(), w.tasks.begin(), w.tasks.end());
    at.obs = flat.size();
    for (uint32_t t : w.tasks) flat.push_back(ps[t]);
    at.cam = flat.size();
    flat.insert(flat.end(), w.chunks.cam.begin(), w.chunks.cam.end());
    at.beg = flat.size();
    flat.insert(flat.end(), w.chunks.beg.begin(), w.chunks.beg.end());
    at.first = flat.size();
    flat.insert(flat.end(), w.chunks.cam_first.begin(), w.chunks.cam_first.end());
    systems.emplace_back(q.cameras, w.pairs, uint32_t(w.chunks.cam.size()), d->sms, all_pairs);
    Cmax = std::max(Cmax, q.cameras);
  }
  auto task_blocks = [&](uint32_t k) {
    return std::max<uint32_t>(1, uint32_t((plans[k].tasks.size() - 1 + 8 * per_warp - 1) / (8 * per_warp)));
  };
  for (uint32_t k : order) {  // largest problems first
    const tba_batch_problem& q = probs[k];
    const SchurLayout& y = systems[k];
    const uint32_t C = q.cameras, P = q.points, M = q.observations;
    const uint64_t n[10] = {1,
                            task_blocks(k),
                            plans[k].chunks.cam.size(),
                            (C + 3) / 4,
                            (std::max(M, C) + 255) / 256,
                            commit_grid(C, P),
                            (12 * uint64_t(C) + 3 * uint64_t(P) + 27 + 255) / 256,
                            C,
                            (y.camera_pairs + 255) / 256,
                            ((y.npairs + y.seg - 1) / y.seg + 7) / 8};
    for (int j = 0; j < 10; j++)
      for (uint32_t b = 0; b < n[j]; b++) lists[j].push_back(make_uint2(k, b));
  }
  const size_t o_flat = L.take<uint32_t>(flat.size());
  size_t o_list[10];
  for (int j = 0; j < 10; j++) o_list[j] = L.take<uint2>(lists[j].size());
  const size_t o_params = L.take<tba::Params>(count), o_schur = L.take<tba::SchurParams>(count),
               o_pcg = L.take<tba::PcgSystem>(count), o_active = L.take<uint32_t>(1);
  // The bit matrices together (zeroed at once), then each problem's workspace.
  size_t bit_words = 0;
  for (uint32_t k = 0; k < count; k++) bit_words += size_t(probs[k].cameras) * ((probs[k].cameras + 31) / 32);
  const size_t o_bits = L.take<uint32_t>(bit_words);
  uint64_t M_all = 0;
  for (uint32_t k = 0; k < count; k++) M_all += probs[k].observations;
  const size_t o_claims = L.take<uint32_t>(whole_check ? M_all : 0), o_bad = L.take<uint32_t>(1),
               o_checks = L.take<tba::CheckProblem>(count);
  struct Work {
    size_t poses, points, cams, pixels, tposes, tpoints, rlim, cmp, cmx, pblk, A, pw, xw, U, Minv, rhs, hcf, scf, chunk, vec, scal, cost, ticket, state, system;
  };
  std::vector<Work> works(count);
  for (uint32_t k = 0; k < count; k++) {
    const size_t C = probs[k].cameras, P = probs[k].points, M = probs[k].observations, m = 6 * C + (shared ? 1 : 0);
    Work& w = works[k];
    w.poses = L.take<double>(12 * C);
    w.points = L.take<double>(3 * P);
    w.cams = L.take<double>(6 * C);
    w.pixels = L.take<double>(2 * M);
    w.tposes = L.take<double>(12 * C);
    w.tpoints = L.take<double>(3 * P);
    w.rlim = L.take<double>(C);
    w.cmp = L.take<uint32_t>(M);
    w.cmx = L.take<double>(2 * M);
    w.pblk = L.take<double>(12 * P);
    w.A = L.take<double>(18 * M);
    w.pw = L.take<double>(6 * C);
    w.xw = L.take<double>(6 * C);
    w.U = L.take<double>(21 * C);
    w.Minv = L.take<double>(36 * C);
    w.rhs = L.take<double>(6 * C);
    w.hcf = L.take<double>(6 * C);
    w.scf = L.take<double>(6 * C);
    w.chunk = L.take<double>(size_t(tba::kCameraPartialsExplicit) * plans[k].chunks.cam.size());
    w.vec = L.take<double>(5 * m);
    w.scal = L.take<double>(size_t(tba::kScalarPartials) * task_blocks(k));
    w.cost = L.take<double>(4 * size_t(task_blocks(k)));
    w.ticket = L.take<uint32_t>(8);
    w.state = L.take<double>(tba::S_WORDS);
    w.system = L.take<char>(systems[k].L.bytes);
  }
  if (d->batch_capacity < L.bytes) {
    if (L.bytes > free_memory(d, L.bytes) + d->batch_capacity) return false;
    if (d->batch_graph) {
      cudaGraphExecDestroy(d->batch_graph);
      d->batch_graph = nullptr;
      d->batch_key.clear();
    }
    grow(d->batch_arena, d->batch_capacity, L.bytes, "GPU BA batch");
  }
  char* a = d->batch_arena;
  auto f64 = [&](size_t off) { return reinterpret_cast<double*>(a + off); };
  auto u32 = [&](size_t off) { return reinterpret_cast<uint32_t*>(a + off); };
  std::vector<tba::Params> params(count);
  std::vector<tba::SchurParams> schur(count);
  std::vector<tba::PcgSystem> pcg(count);
  size_t bits = 0;
  for (uint32_t k = 0; k < count; k++) {
    const tba_batch_problem& q = probs[k];
    const Work& w = works[k];
    const Place& at = places[k];
    const size_t C = q.cameras, P = q.points, M = q.observations;
    tba::Params& p = params[k];
    tba::SchurParams& y = schur[k];
    tba::PcgSystem& c = pcg[k];
    p = tba::Params{};
    p.C = q.cameras;
    p.P = q.points;
    p.M = q.observations;
    p.m = 6 * q.cameras + (shared ? 1 : 0);
    p.anchor = q.anchor;
    p.scale_view = q.scale_view;
    p.shared = shared;
    p.huber = bc->huber;
    p.tol = p.tol_inner = bc->cg_tolerance;
    p.stall = bc->stall_tolerance;
    const uint32_t* act = index + q.index_offset + 3 * M + P + C + 2;
    uint32_t fixed = 0;
    for (size_t j = 0; j < C; j++) fixed += act[j] == 0;
    p.normalize_scale = fixed == 1;
    p.packed = f64(o_scene) + q.scene_offset;
    p.poses = f64(w.poses);
    p.points = f64(w.points);
    p.cams = f64(w.cams);
    p.pixels = f64(w.pixels);
    p.tposes = f64(w.tposes);
    p.tpoints = f64(w.tpoints);
    const uint32_t* x = u32(o_index) + q.index_offset;
    p.obs_camera = x;
    p.obs_point = x + M;
    p.point_start = x + 2 * M;
    p.camera_start = p.point_start + P + 1;
    p.camera_obs = p.camera_start + C + 1;
    p.active = p.camera_obs + M;
    p.tasks = u32(o_flat) + at.tasks;
    p.task_obs = u32(o_flat) + at.obs;
    p.ntasks = uint32_t(plans[k].tasks.size() - 1);
    p.chunk_cam = u32(o_flat) + at.cam;
    p.chunk_beg = u32(o_flat) + at.beg;
    p.cam_chunk = u32(o_flat) + at.first;
    p.nchunks = uint32_t(plans[k].chunks.cam.size());
    p.task_blocks = task_blocks(k);
    p.commit_blocks = commit_grid(q.cameras, q.points);
    p.rlim = f64(w.rlim);
    p.cm_point = u32(w.cmp);
    p.cm_pixel = f64(w.cmx);
    p.pblk = f64(w.pblk);
    p.Mpad = uint32_t((M + 31) / 32 * 32);
    p.factored = p.schur = 1;
    p.A = f64(w.A);
    p.camScf = f64(w.scf);
    p.pw = f64(w.pw);
    p.xw = f64(w.xw);
    p.camU = f64(w.U);
    p.camMinv = f64(w.Minv);
    p.camRhs = f64(w.rhs);
    p.camHcf = f64(w.hcf);
    p.chunk_part = f64(w.chunk);
    p.x = f64(w.vec);
    p.r = p.x + p.m;
    p.p = p.r + p.m;
    p.Sp = p.p + p.m;
    p.z = p.Sp + p.m;
    p.scal_part = f64(w.scal);
    p.cost_part = f64(w.cost);
    p.ticket = u32(w.ticket);
    p.state = f64(w.state);
    p.output = f64(o_out) + q.output_offset;
    y = tba::SchurParams{};
    c = tba::PcgSystem{};
    systems[k].bind(a + w.system, y, c);
    y.bits = u32(o_bits) + bits;
    bits += size_t(C) * y.bwords;
    bind_problem(p, y, c);  // (one block a problem: nothing waits)
  }
  cudaStream_t s = d->stream;
  auto up = [&](size_t off, const void* src, size_t bytes) {
    if (bytes) CUDA_TRY(cudaMemcpyAsync(a + off, src, bytes, cudaMemcpyHostToDevice, s));
    h2d += bytes;
  };
  CUDA_TRY(cudaEventRecord(begun, s));
  up(o_scene, scene, scene_len * sizeof(double));
  up(o_index, index, index_len * sizeof(uint32_t));
  up(o_flat, flat.data(), flat.size() * sizeof(uint32_t));
  for (int j = 0; j < 10; j++) up(o_list[j], lists[j].data(), lists[j].size() * sizeof(uint2));
  up(o_params, params.data(), count * sizeof(tba::Params));
  up(o_schur, schur.data(), count * sizeof(tba::SchurParams));
  up(o_pcg, pcg.data(), count * sizeof(tba::PcgSystem));
  std::vector<tba::CheckProblem> checks(count);
  if (whole_check) {
    uint64_t claims = 0;
    for (uint32_t k = 0; k < count; k++) {
      const tba::Params& p = params[k];
      checks[k] = tba::CheckProblem{p.C, p.P, p.M, (std::max(p.M, p.C) + 255) / 256, p.obs_camera, p.packed, u32(o_claims) + claims};
      claims += p.M;
    }
    up(o_checks, checks.data(), count * sizeof(tba::CheckProblem));
  }
  CUDA_TRY(cudaEventRecord(uploaded, s));
  uint32_t launches = 0;
  if (whole_check) {
    CUDA_TRY(cudaMemsetAsync(a + o_claims, 0, M_all * sizeof(uint32_t), s));
    CUDA_TRY(cudaMemsetAsync(a + o_bad, 0, sizeof(uint32_t), s));
    tba::launch_check_batch(reinterpret_cast<const tba::CheckProblem*>(a + o_checks), reinterpret_cast<const uint2*>(a + o_list[4]),
                            uint32_t(lists[4].size()), u32(o_bad), s);
    launches++;
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaMemcpyAsync(d->pinned, a + o_bad, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaStreamSynchronize(s));
    if (*reinterpret_cast<const uint32_t*>(d->pinned) != 0) {
      (*whole_check)();
      throw Fail{TBA_ERROR_INTERNAL, "GPU BA batch checks disagree"};
    }
  }

  struct Key {
    tba::ManyLists many;
    tba::SchurLists schur;
    tba::PcgMany pcg;
    uint32_t count, limit;
  } key;
  std::memset(&key, 0, sizeof key);
  auto list = [&](auto& to, int j) {
    to.work = reinterpret_cast<const uint2*>(a + o_list[j]);
    to.blocks = uint32_t(lists[j].size());
  };
  key.many.params = reinterpret_cast<const tba::Params*>(a + o_params);
  key.many.active = u32(o_active);
  key.many.count = count;
  key.many.shared = shared;
  list(key.many.one, 0);
  list(key.many.task, 1);
  list(key.many.chunk, 2);
  list(key.many.finish, 3);
  list(key.many.setup, 4);
  list(key.many.commit, 5);
  list(key.many.pack, 6);
  key.schur.params = reinterpret_cast<const tba::SchurParams*>(a + o_schur);
  key.schur.max_cameras = Cmax;
  list(key.schur.one, 0);
  list(key.schur.chunk, 2);
  list(key.schur.camera, 7);
  list(key.schur.pairs, 8);
  list(key.schur.sums, 9);
  key.pcg.systems = reinterpret_cast<const tba::PcgSystem*>(a + o_pcg);
  key.pcg.work = key.many.one.work;
  key.count = count;
  // (a mixed request: the budgets of the mixed form's run and its restart)
  key.limit = bc->max_cg * (bc->precision == TBA_PRECISION_MIXED ? 2 : 1);
  CUDA_TRY(cudaMemsetAsync(a + o_bits, 0, bit_words * sizeof(uint32_t), s));
  launches += tba::launch_many_begin(key.many, s);
  launches += tba::schur_launch_many_structure(key.schur, s);
  launches += tba::pcg_launch_many_plan(key.pcg, count, Cmax, s);
  CUDA_TRY(cudaGetLastError());
  uint32_t per_iteration = 0;
  auto iteration = [&]() {
    per_iteration = tba::launch_many_linearize(key.many, s);
    per_iteration += tba::schur_launch_many_values(key.schur, s);
    const cudaError_t e = tba::launch_many_pcg(key.pcg, count, shared, key.limit, s);
    per_iteration += 1 + tba::launch_many_update(key.many, s);
    return e;
  };
  const char* bytes = reinterpret_cast<const char*>(&key);
  rep.replayed = d->window_graph && d->window_key.size() == sizeof key && std::memcmp(d->window_key.data(), bytes, sizeof key) == 0;
  if (!rep.replayed) {
    if (d->window_graph) {
      CUDA_TRY(cudaGraphExecDestroy(d->window_graph));
      d->window_graph = nullptr;
    }
    cudaGraph_t graph = nullptr;
    CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    const cudaError_t e1 = iteration();
    const cudaError_t e2 = cudaGetLastError(), e3 = cudaStreamEndCapture(s, &graph);
    CUDA_TRY(e1);
    CUDA_TRY(e2);
    CUDA_TRY(e3);
    const cudaError_t e4 = cudaGraphInstantiate(&d->window_graph, graph, 0);
    cudaGraphDestroy(graph);
    if (e4 != cudaSuccess) d->window_graph = nullptr;
    CUDA_TRY(e4);
    d->window_key.assign(bytes, bytes + sizeof key);
  } else {
    per_iteration = 3 + 2 + 1 + 4;
  }
  // Iterations are issued one ahead of the last one known to have left active problems.
  uint32_t* active = reinterpret_cast<uint32_t*>(d->pinned);
  *active = 1;
  cudaEvent_t done[2] = {event(d, 6), event(d, 7)};
  for (uint32_t it = 0; it < bc->iterations; it++) {
    if (it >= 2) {
      CUDA_TRY(cudaEventSynchronize(done[it & 1]));
      if (*reinterpret_cast<volatile uint32_t*>(active) == 0) break;
    }
    CUDA_TRY(cudaGraphLaunch(d->window_graph, s));
    launches += per_iteration;
    CUDA_TRY(cudaMemcpyAsync(active, key.many.active, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaEventRecord(done[it & 1], s));
  }
  launches += tba::launch_many_pack(key.many, s);
  CUDA_TRY(cudaGetLastError());
  // The host arrays above stay until their copies are done.
  CUDA_TRY(cudaEventSynchronize(uploaded));
  rep.shape = tba::kBatchGridShape;
  rep.threads = tba::kBatchGridThreads;
  rep.blocks = key.many.task.blocks;
  rep.launches = launches;
  dout_of = f64(o_out);
  return true;
}

// Whether the windows' PCG steps cost less on the systems, one block a window, than on the block solver: there
// 14 us and 11.5 ns an observation; here 5 us, 80 ns a camera and 4.2 ns a block of S, or, where the S of the windows
// in flight (one an SM) do not stay in the L2, their bytes from DRAM.  The blocks are the bound's, or where that
// says no, those that a window's camera pairs spread over.  Whole batches, six iterations, every camera sharing
// points with any other, block solver and systems, ms: 1 window of 60 cameras / 2,000 observations 8.5 and 4.8,
// 100 / 3,000 12.1 and 10.4, 144 / 3,000 12.5 and 13.8, 144 / 25,000 47.6 and 18.4; 148 windows of 60 / 2,000 with the
// focal unknown 11.0 and 13.8, of 144 / 3,000 16.1 and 30.8.
bool systems_pay(const tba_batch_problem* probs, uint32_t count, const std::vector<WindowPlan>& plans,
                 const uint32_t* index, int sms) {
  double product = 0, cameras = 0, bound = 0;
  for (uint32_t k = 0; k < count; k++) {
    product += 14 + 11.5e-3 * double(probs[k].observations);
    cameras += 5 + 0.08 * probs[k].cameras;
    bound += double(schur_block_bound(probs[k].cameras, plans[k].pairs));
  }
  const auto pay = [&](double blocks) {
    // (the windows in flight read their systems together, at 4.5 TB/s)
    const double flight = 288 * blocks * std::min(1.0, double(sms) / count);
    return cameras + std::max(4.2e-3 * blocks, flight > 100e6 ? flight / 4.5e6 * count : 0) < product;
  };
  if (pay(bound)) return true;
  double found = 0, of = 0;  // at most eight of the windows tell for all
  for (uint32_t k = 0; k < count; k += (count + 7) / 8) {
    const tba_batch_problem& q = probs[k];
    const double most = double(schur_block_bound(q.cameras, plans[k].pairs));
    found += std::min(most, spread_blocks(q.cameras, q.points, q.observations, index + q.index_offset));
    of += most;
  }
  return pay(bound * found / of);
}

void solve_batch(tba_device* d, const tba_batch_control* bc, const tba_batch_problem* probs, uint32_t count,
                 const double* scene, size_t scene_len, const uint32_t* index, size_t index_len, double* output,
                 size_t output_len, tba_batch_report* report) {
  const auto wall0 = std::chrono::steady_clock::now();
  const bool shared = bc->shared_focal != 0, mixed = bc->precision == TBA_PRECISION_MIXED;
  const uint32_t max_cams = tba::batch_max_cameras();
  uint32_t Cmax = 2;
  std::vector<uint32_t> tasks;
  std::vector<uint64_t> task_first(count), task_count(count);
  // Each problem is checked and scheduled on its own; the problems are spread over host threads and
  // the failure reported is the one of the first failing problem, as a loop in order would report.
  std::vector<WindowPlan> plans(count);
  const bool auto_shape = bc->schedule == 0, grid_forced = bc->schedule == uint32_t(tba::kBatchGridShape) + 1;
  uint64_t M_all = 0;
  for (uint32_t k = 0; k < count; k++) M_all += probs[k].observations;
  const uint32_t chunk = std::min<uint32_t>(1024, chunk_size(M_all, d->sms));
  std::mutex fail_mu;
  uint32_t fail_at = UINT32_MAX;
  Fail first_fail{TBA_OK, ""};
  // On the grid kernels the O(M) checks run on the device: the host makes the others here, and repeats all
  // of them, for the message, where one of either kind fails.
  std::vector<uint8_t> suspect(count, 0);
  auto check_problems = [&](bool whole) {
    parallel_ranges(count, 2, [&](uint64_t b, uint64_t e, unsigned) {
      for (uint64_t k = b; k < e; k++) {
        try {
          const tba_batch_problem& q = probs[k];
          const tba_control c = batch_problem_control(bc, q);
          check_control(&c);
          if (q.reserved != 0) argument("Invalid GPU BA batch: reserved field must be 0");
          if (q.cameras > max_cams)
            argument("Batched GPU BA problem has " + std::to_string(q.cameras) +
                     " cameras; the block solver takes at most " + std::to_string(max_cams));
          if (uint64_t(3) * q.observations + q.points + 2ull * q.cameras + 2 > 0xffffffffull)
            argument("GPU BA scene dimensions exceed integer index bounds");
          if (q.scene_offset > scene_len || scene_len - q.scene_offset < tba_scene_size(&c))
            argument("Invalid GPU BA batch: a scene lies outside the scene array");
          if (q.index_offset > index_len || index_len - q.index_offset < tba_index_size(&c))
            argument("Invalid GPU BA batch: an index lies outside the index array");
          if (q.output_offset > output_len || output_len - q.output_offset < tba_output_size(&c))
            argument("Invalid GPU BA batch: a result record lies outside the output array");
          if (whole) {
            check_index(&c, index + q.index_offset);
            check_scene(&c, scene + q.scene_offset, tba_scene_size(&c));
          } else {
            const HostChecks h = host_checks(&c, index + q.index_offset, scene + q.scene_offset);
            if (h.point_ends || h.camera_ends || h.camera_offsets || h.activity || h.camera_bounds) {
              suspect[k] = 1;
              continue;
            }
          }
          if (!plans[k].tasks.empty()) continue;  // planned before the whole check
          const uint32_t* ps = index + q.index_offset + 2 * size_t(q.observations);
          plans[k].tasks = build_tasks(ps, q.points);
          if (auto_shape || grid_forced) {
            plans[k].chunks = build_chunks(ps + q.points + 1, q.cameras, chunk);
            plans[k].pairs = count_pairs(ps, q.points).pairs;
          }
        } catch (const Fail& f) {
          std::lock_guard<std::mutex> lock(fail_mu);
          if (k < fail_at) {
            fail_at = uint32_t(k);
            first_fail = f;
          }
          return;
        }
      }
    });
    if (fail_at != UINT32_MAX) throw first_fail;
  };
  bool checked = false;
  auto check_whole = [&] {
    if (!checked) check_problems(true);
    checked = true;
  };
  if ((auto_shape || grid_forced) && M_all >= kDeviceCheckMin) {
    try {
      check_problems(false);
    } catch (const Fail&) {
      fail_at = UINT32_MAX;
      check_whole();
      throw;
    }
    if (std::find(suspect.begin(), suspect.end(), 1) != suspect.end()) check_whole();
  } else {
    check_whole();
  }
  for (uint32_t k = 0; k < count; k++) {
    const std::vector<uint32_t>& t = plans[k].tasks;
    task_first[k] = tasks.size();
    task_count[k] = t.size() - 1;
    tasks.insert(tasks.end(), t.begin(), t.end());
    Cmax = std::max(Cmax, probs[k].cameras);
  }
  // Result records must not overlap: the device writes each one whole.
  std::vector<uint32_t> by_out(count);
  std::iota(by_out.begin(), by_out.end(), 0u);
  std::sort(by_out.begin(), by_out.end(), [&](uint32_t a, uint32_t b) { return probs[a].output_offset < probs[b].output_offset; });
  for (uint32_t j = 1; j < count; j++) {
    const tba_batch_problem& prev = probs[by_out[j - 1]];
    const tba_control pc = batch_problem_control(bc, prev);
    if (prev.output_offset + tba_output_size(&pc) > probs[by_out[j]].output_offset) {
      check_whole();
      argument("Invalid GPU BA batch: result records overlap");
    }
  }
  // Largest problems first (longest-processing-time order for the persistent blocks).
  std::vector<uint32_t> order(count);
  std::iota(order.begin(), order.end(), 0u);
  std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) {
    return uint64_t(probs[a].observations) * probs[a].cameras > uint64_t(probs[b].observations) * probs[b].cameras;
  });

  cudaStream_t s = d->stream;
  cudaEvent_t e0 = event(d, 0), e1 = event(d, 1), e2 = event(d, 2), e3 = event(d, 3);
  uint64_t h2d = 0;
  double tune_ms = 0;
  BatchReport ran;
  // Download of the result records, merged into contiguous runs, and the report.
  auto finish = [&](const double* dout) {
    CUDA_TRY(cudaEventRecord(e2, s));
    uint64_t d2h = 0;
    for (uint32_t j = 0; j < count;) {
      const tba_batch_problem& q0 = probs[by_out[j]];
      const size_t begin = q0.output_offset;
      tba_control c0 = batch_problem_control(bc, q0);
      size_t end = begin + tba_output_size(&c0);
      uint32_t k = j + 1;
      while (k < count && probs[by_out[k]].output_offset == end) {
        const tba_control ck = batch_problem_control(bc, probs[by_out[k]]);
        end += tba_output_size(&ck);
        k++;
      }
      CUDA_TRY(cudaMemcpyAsync(output + begin, dout + begin, (end - begin) * sizeof(double), cudaMemcpyDeviceToHost, s));
      d2h += (end - begin) * sizeof(double);
      j = k;
    }
    CUDA_TRY(cudaEventRecord(e3, s));
    CUDA_TRY(cudaStreamSynchronize(s));
    if (report) {
      std::memset(report, 0, sizeof *report);
      float ms = 0;
      CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
      report->upload_ms = ms;
      CUDA_TRY(cudaEventElapsedTime(&ms, e1, e2));
      report->solve_ms = ms;
      CUDA_TRY(cudaEventElapsedTime(&ms, e2, e3));
      report->download_ms = ms;
      report->tune_ms = tune_ms;
      report->h2d_bytes = h2d;
      report->d2h_bytes = d2h;
      for (uint32_t k = 0; k < count; k++) {
        const tba_batch_problem& q = probs[k];
        const double* st = output + q.output_offset + 12 * size_t(q.cameras) + 3 * size_t(q.points);
        report->lm_iterations += uint64_t(st[tba::S_ACCEPTED] + st[tba::S_REJECTED]);
        report->cg_iterations += uint64_t(st[tba::S_CG_STEPS]);
      }
      report->problems = count;
      report->schedule = uint32_t(ran.shape);
      report->threads = ran.threads;
      report->blocks = ran.blocks;
      report->graph_replayed = ran.replayed ? 1 : 0;
      report->kernel_launches = ran.launches;
      report->form = ran.mixed ? TBA_PRECISION_MIXED : TBA_PRECISION_FP64;
      report->wall_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - wall0).count();
    }
  };
  // The grid kernels unless another shape is asked for.  They form each reduced system, at a cost that
  // grows with the pairs of observations of a point; beyond tracks of about 64 that is more than the
  // block solver's passes over the observations, and they need the memory for them.  Nor are they taken
  // where the systems are large for what the windows observe.
  if (auto_shape || grid_forced) {
    uint64_t pairs = 0;
    bool fits = true;
    for (uint32_t k = 0; k < count; k++) {
      pairs += plans[k].pairs;
      fits = fits && plans[k].pairs < 0x7fffffffull;
    }
    double* dout = nullptr;
    const std::function<void()> whole = check_whole;
    if (fits && (grid_forced || (pairs <= 32 * M_all && systems_pay(probs, count, plans, index, d->sms))) &&
        batch_on_grid(d, bc, probs, count, plans, order, scene, scene_len, index, index_len, output_len, e1, e0, ran, dout, h2d,
                      checked ? nullptr : static_cast<const std::function<void()>*>(&whole))) {
      finish(dout);
      return;
    }
    check_whole();
    if (grid_forced) throw Fail{TBA_ERROR_BUDGET, "GPU BA batch needs more device memory than the working budget"};
  }

  // Device layout: the caller's arrays as they are, then the schedule and the workspace.
  Layout L;
  const size_t factor_size = mixed ? 4 : 8;
  const size_t o_scene = L.take<double>(scene_len), o_index = L.take<uint32_t>(index_len),
               o_out = L.take<double>(output_len), o_tasks = L.take<uint32_t>(tasks.size()),
               o_desc = L.take<tba::BatchProblem>(count), o_desc64 = L.take<tba::BatchProblem>(mixed ? count : 0),
               o_order = L.take<uint32_t>(count),
               o_queue = L.take<uint32_t>(4);
  std::vector<size_t> o_tp(count), o_pb(count), o_F(count), o_F64(count);
  uint64_t M_total = 0;
  for (uint32_t k = 0; k < count; k++) {
    const tba_batch_problem& q = probs[k];
    const size_t Mpad = (size_t(q.observations) + 31) / 32 * 32;
    o_tp[k] = L.take<double>(3 * size_t(q.points));
    o_pb[k] = L.take<double>(12 * size_t(q.points));
    o_F[k] = L.take<char>(tba::kFactors * Mpad * factor_size);
    o_F64[k] = L.take<char>(mixed ? tba::kFactors * Mpad * sizeof(double) : 0);  // the mixed form's FP64 copy
    M_total += q.observations;
  }
  if (d->batch_capacity < L.bytes) {
    if (d->batch_graph) {
      cudaGraphExecDestroy(d->batch_graph);
      d->batch_graph = nullptr;
      d->batch_key.clear();
    }
    if (d->batch_arena) CUDA_TRY(cudaFree(d->batch_arena));
    d->batch_arena = nullptr;
    d->batch_capacity = 0;
    const size_t free_bytes = free_memory(d, L.bytes);
    if (L.bytes > free_bytes)
      throw Fail{TBA_ERROR_BUDGET, "GPU BA batch needs " + std::to_string(L.bytes) +
                                       " bytes of device memory, more than the working budget of " +
                                       std::to_string(free_bytes) + " bytes"};
    CUDA_TRY(cudaMalloc(&d->batch_arena, L.bytes));
    d->batch_capacity = L.bytes;
  }
  char* a = d->batch_arena;
  const double* dscene = reinterpret_cast<const double*>(a + o_scene);
  const uint32_t* dindex = reinterpret_cast<const uint32_t*>(a + o_index);
  double* dout = reinterpret_cast<double*>(a + o_out);
  const uint32_t* dtasks = reinterpret_cast<const uint32_t*>(a + o_tasks);
  std::vector<tba::BatchProblem> desc(count);
  for (uint32_t k = 0; k < count; k++) {
    const tba_batch_problem& q = probs[k];
    tba::BatchProblem& b = desc[k];
    const uint32_t C = q.cameras, P = q.points, M = q.observations;
    b.C = C;
    b.P = P;
    b.M = M;
    b.ntasks = uint32_t(task_count[k]);
    b.anchor = q.anchor;
    b.scale_view = q.scale_view;
    const uint32_t* act = index + q.index_offset + 3 * size_t(M) + P + C + 2;
    uint32_t fixed = 0;
    for (uint32_t c = 0; c < C; c++) fixed += act[c] == 0;
    b.normalize_scale = fixed == 1;
    b.Mpad = uint32_t((size_t(M) + 31) / 32 * 32);
    const double* s = dscene + q.scene_offset;
    b.poses0 = s;
    b.points0 = s + 12 * size_t(C);
    b.cams = s + 12 * size_t(C) + 3 * size_t(P);
    b.pixels = s + 18 * size_t(C) + 3 * size_t(P);
    const uint32_t* x = dindex + q.index_offset;
    b.obs_camera = x;
    b.obs_point = x + M;
    b.point_start = x + 2 * size_t(M);
    b.camera_start = b.point_start + P + 1;
    b.camera_obs = b.camera_start + C + 1;
    b.active = b.camera_obs + M;
    b.tasks = dtasks + task_first[k];
    b.tpoints = reinterpret_cast<double*>(a + o_tp[k]);
    b.pblk = reinterpret_cast<double*>(a + o_pb[k]);
    b.F = a + o_F[k];
    b.F64 = mixed ? reinterpret_cast<double*>(a + o_F64[k]) : nullptr;
    b.output = dout + q.output_offset;
    b.points = b.output + 12 * size_t(C);
  }

  tba::BatchArgs args{};
  args.problems = reinterpret_cast<const tba::BatchProblem*>(a + o_desc);
  args.order = reinterpret_cast<const uint32_t*>(a + o_order);
  args.queue = reinterpret_cast<uint32_t*>(a + o_queue);
  args.count = count;
  args.Cmax = Cmax;
  args.iterations = bc->iterations;
  args.max_cg = bc->max_cg;
  args.huber = bc->huber;
  args.tol = bc->cg_tolerance;
  args.tol_inner = mixed ? std::max(bc->cg_tolerance, 1e-6) : bc->cg_tolerance;
  args.stall = bc->stall_tolerance;
  const size_t smem = tba::batch_smem_bytes(Cmax);

  auto up = [&](size_t off, const void* src, size_t bytes) {
    if (bytes) CUDA_TRY(cudaMemcpyAsync(a + off, src, bytes, cudaMemcpyHostToDevice, s));
    h2d += bytes;
  };
  CUDA_TRY(cudaEventRecord(e0, s));
  up(o_scene, scene, scene_len * sizeof(double));
  up(o_index, index, index_len * sizeof(uint32_t));
  up(o_tasks, tasks.data(), tasks.size() * sizeof(uint32_t));
  up(o_desc, desc.data(), desc.size() * sizeof(tba::BatchProblem));
  up(o_order, order.data(), order.size() * sizeof(uint32_t));
  // A mixed request may also run as the FP64 form (the tuner's policy choice below): the same
  // problems with their factors in the FP64 region and no FP32 copy.
  tba::BatchArgs args64 = args;
  if (mixed) {
    std::vector<tba::BatchProblem> desc64 = desc;
    for (tba::BatchProblem& b : desc64) {
      b.F = b.F64;
      b.F64 = nullptr;
    }
    up(o_desc64, desc64.data(), desc64.size() * sizeof(tba::BatchProblem));
    args64.problems = reinterpret_cast<const tba::BatchProblem*>(a + o_desc64);
    args64.tol_inner = bc->cg_tolerance;
  }
  CUDA_TRY(cudaEventRecord(e1, s));

  auto blocks_of = [&](int shape, bool form_mixed) {
    const int per_sm = tba::batch_blocks_per_sm(shape, shared, form_mixed, smem);
    return std::min<int>(int(count), per_sm * d->sms);
  };
  // The launch shape, and for a mixed request the form: forced, cached, or tuned now by one timed
  // LM iteration of the whole batch per shape (the trial launches write only the workspace and the
  // device copy of the results).  A mixed request tries the FP64 form too and keeps it when it is
  // faster: on small windows the FP32 product saves less than the FP64 refinement of each PCG
  // solution costs.  The result is the FP64 form's, which the mixed form only approximates.
  int shape = -1;
  bool run_mixed = mixed;
  if (bc->schedule > 0) {
    shape = int(bc->schedule) - 1;
    if (shape >= tba::kBatchShapes) argument("Invalid GPU BA batch schedule");
  } else {
    int lg = 0;
    while ((uint64_t(1) << (lg + 1)) <= std::max<uint64_t>(1, M_total)) lg++;
    const std::string key = std::to_string(shared) + "/" + std::to_string(mixed) + "/" + std::to_string(Cmax) + "/" +
                            std::to_string(lg) + "/" + std::to_string(count);
    auto hit = d->tuned.find(key);
    if (hit != d->tuned.end()) {
      shape = hit->second % tba::kBatchShapes;
      run_mixed = mixed && hit->second < tba::kBatchShapes;
    } else {
      const auto t0 = std::chrono::steady_clock::now();
      cudaEvent_t ta = event(d, 4), tb = event(d, 5);
      // One timed launch of the batch in one form and shape; -1 when the shape does not fit.
      auto trial_ms = [&](int k, bool form_mixed, uint32_t iterations) -> float {
        const int blocks = blocks_of(k, form_mixed);
        if (blocks <= 0) return -1;
        tba::BatchArgs trial = form_mixed || !mixed ? args : args64;
        trial.iterations = iterations;
        CUDA_TRY(cudaMemsetAsync(trial.queue, 0, sizeof(uint32_t), s));
        CUDA_TRY(cudaEventRecord(ta, s));
        CUDA_TRY(tba::launch_batch(k, shared, form_mixed, trial, blocks, smem, s));
        CUDA_TRY(cudaEventRecord(tb, s));
        CUDA_TRY(cudaStreamSynchronize(s));
        float ms = 0;
        CUDA_TRY(cudaEventElapsedTime(&ms, ta, tb));
        return ms;
      };
      // Each form's shape by one LM iteration per shape; for a mixed request the two forms' best
      // shapes then run the whole solve once each (one LM iteration does not show the refinement's
      // share), and the faster form is kept.
      int best_shape[2] = {-1, -1};
      for (int form = 0; form < (mixed ? 2 : 1); form++) {
        const bool form_mixed = mixed && form == 0;
        float best = 0;
        for (int k = 0; k < tba::kBatchShapes; k++) {
          const float ms = trial_ms(k, form_mixed, std::min<uint32_t>(args.iterations, 1));
          if (ms >= 0 && (best_shape[form] < 0 || ms < best)) {
            best = ms;
            best_shape[form] = k;
          }
        }
      }
      shape = best_shape[0];
      run_mixed = mixed;
      if (mixed && best_shape[0] >= 0 && best_shape[1] >= 0 && args.iterations > 1) {
        const float ms_mixed = trial_ms(best_shape[0], true, args.iterations);
        const float ms_fp64 = trial_ms(best_shape[1], false, args.iterations);
        if (ms_fp64 < ms_mixed) {
          shape = best_shape[1];
          run_mixed = false;
        }
      } else if (shape < 0) {
        shape = best_shape[1];
        run_mixed = false;
      }
      if (shape < 0) throw Fail{TBA_ERROR_INTERNAL, "no launch shape of the batched solver fits the device"};
      d->tuned[key] = shape + (mixed && !run_mixed ? tba::kBatchShapes : 0);
      tune_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }
  }
  if (!run_mixed) args = args64;  // (args64 == args for an FP64 request)
  const int blocks = blocks_of(shape, run_mixed);
  if (blocks <= 0) throw Fail{TBA_ERROR_INTERNAL, "the batched solver's launch shape does not fit the device"};

  // One persistent launch, captured once in a CUDA graph and replayed while its arguments stay.
  std::vector<char> key(sizeof args + 3 * sizeof(int) + sizeof(size_t));
  {
    const int ints[3] = {shape, blocks, int(shared) | (int(run_mixed) << 1)};
    std::memcpy(key.data(), &args, sizeof args);
    std::memcpy(key.data() + sizeof args, ints, sizeof ints);
    std::memcpy(key.data() + sizeof args + sizeof ints, &smem, sizeof smem);
  }
  bool replayed = true;
  if (!d->batch_graph || d->batch_key != key) {
    replayed = false;
    if (d->batch_graph) {
      CUDA_TRY(cudaGraphExecDestroy(d->batch_graph));
      d->batch_graph = nullptr;
    }
    cudaGraph_t graph = nullptr;
    CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    cudaError_t e1c = cudaMemsetAsync(args.queue, 0, sizeof(uint32_t), s);
    cudaError_t e2c = e1c == cudaSuccess ? tba::launch_batch(shape, shared, run_mixed, args, blocks, smem, s) : e1c;
    cudaError_t e3c = cudaStreamEndCapture(s, &graph);
    CUDA_TRY(e2c);
    CUDA_TRY(e3c);
    cudaError_t ei = cudaGraphInstantiate(&d->batch_graph, graph, 0);
    cudaGraphDestroy(graph);
    CUDA_TRY(ei);
    d->batch_key = key;
  }
  CUDA_TRY(cudaGraphLaunch(d->batch_graph, s));
  ran.shape = shape;
  ran.threads = uint32_t(tba::batch_shape(shape).threads);
  ran.blocks = uint32_t(blocks);
  ran.launches = 2;
  ran.replayed = replayed;
  ran.mixed = run_mixed;
  finish(dout);
}

// ---- the adjoint ---------------------------------------------------------------------------------

// `checks`: the host's part of the checks, whose O(M) part then runs on the device; null when all are done.
void solve_vjp(tba_device* d, const tba_vjp_control* vc, const HostChecks* checks, const double* scene,
               const uint32_t* index, const double* cotangent, double* pixels_bar, double* intrinsics_bar,
               double* solution, tba_vjp_report* report) {
  const auto wall0 = std::chrono::steady_clock::now();
  const uint32_t C = vc->cameras, P = vc->points, M = vc->observations;
  const uint32_t* active = index + 3 * size_t(M) + P + C + 2;
  uint32_t fixed = 0;
  for (uint32_t c = 0; c < C; c++) fixed += active[c] == 0;
  tba::AdjParams A{};
  A.C = C;
  A.P = P;
  A.M = M;
  A.anchor = vc->anchor;
  A.scale_view = vc->scale_view;
  A.normalize_scale = fixed == 1;
  A.huber = vc->huber;
  A.tol = vc->cg_tolerance;
  // Warp tasks of the one-pass Schur product (whole points, at most 32 observations each).
  const std::vector<uint32_t> tasks = build_tasks(index + 2 * size_t(M), P);
  std::vector<uint32_t> task_obs(tasks.size());
  for (size_t t = 0; t < tasks.size(); t++) task_obs[t] = index[2 * size_t(M) + tasks[t]];
  A.ntasks = uint32_t(tasks.size() - 1);
  A.prod_blocks = C <= tba::adj_one_pass_max_cameras()
                      ? std::max<uint32_t>(1, std::min<uint32_t>(tba::adj_product_blocks_per_sm(C) * uint32_t(d->sms),
                                                                 (A.ntasks + 7) / 8))
                      : 0;
  A.prod_copies = tba::adj_product_copies(C);
  // The explicit reduced system in place of the product over the cross blocks, where it costs less and
  // fits the device.  (With one variable camera there is nothing to gain: its preconditioner is the inverse, and
  // a call of two cameras took 0.21 ms instead of 0.19 for the system's structure.)
  const Tracks tracks = survey(C, P, M, index);
  const uint64_t npairs = tracks.pairs;
  bool schur = C - fixed > 1 && prefer_schur(C, M, Tracks{npairs, 0, tracks.spread}, vc->max_cg, 64, vc->max_cg, false);
  Chunks chunks;
  if (checks && (checks->camera_ends || checks->camera_offsets)) schur = false;  // no chunks; the checks will fail
  if (schur) chunks = build_chunks(index + 2 * size_t(M) + P + 1, C, chunk_size(M, d->sms));
  const uint32_t nchunks = uint32_t(chunks.cam.size());
  Layout L;
  const size_t o_poses = L.take<double>(12 * size_t(C)), o_points = L.take<double>(3 * size_t(P)),
               o_cams = L.take<double>(6 * size_t(C)), o_pixels = L.take<double>(2 * size_t(M)),
               o_index = L.take<uint32_t>(3 * size_t(M) + P + 2 * size_t(C) + 2),
               o_hcp = L.take<double>(18 * size_t(M)), o_hcc = L.take<double>(21 * size_t(M)),
               o_hpp = L.take<double>(6 * size_t(M)), o_gc = L.take<double>(6 * size_t(M)),
               o_gp = L.take<double>(3 * size_t(M)), o_vinv = L.take<double>(6 * size_t(P)),
               o_bp = L.take<double>(3 * size_t(P)), o_lp = L.take<double>(3 * size_t(P)),
               o_yp = L.take<double>(3 * size_t(P)), o_U = L.take<double>(21 * size_t(C)),
               o_minv = L.take<double>(36 * size_t(C)), o_bc = L.take<double>(6 * size_t(C)),
               o_vec = L.take<double>(5 * 6 * size_t(C)), o_cot = L.take<double>(6 * size_t(C) + 3 * size_t(P)),
               o_gcot = L.take<double>(12 * size_t(C) + 3 * size_t(P)), o_ybar = L.take<double>(2 * size_t(M)),
               o_state = L.take<double>(tba::A_WORDS), o_tposes = L.take<double>(12 * size_t(C)),
               o_tpoints = L.take<double>(3 * size_t(P)), o_tobs = L.take<uint32_t>(task_obs.size()),
               o_part = L.take<double>(size_t(A.prod_blocks) * 6 * C);
  const size_t product_only = L.bytes;
  const size_t o_root = L.take<double>(schur ? 6 * size_t(P) : 0), o_ccam = L.take<uint32_t>(nchunks),
               o_cbeg = L.take<uint32_t>(nchunks + 1), o_cfirst = L.take<uint32_t>(schur ? C + 1 : 0);
  const SchurLayout Q(schur ? C : 0, schur ? npairs : 0, nchunks, d->sms);
  if (schur && !memory_for(d, L.bytes, Q.L.bytes)) schur = false;
  make_room(d, schur ? L.bytes : product_only, schur ? Q.L.bytes : 0, "GPU BA adjoint");
  char* a = d->arena;
  auto D = [&](size_t off) { return reinterpret_cast<double*>(a + off); };
  A.poses = D(o_poses);
  A.points = D(o_points);
  A.cams = D(o_cams);
  A.pixels = D(o_pixels);
  uint32_t* dindex = reinterpret_cast<uint32_t*>(a + o_index);
  A.obs_camera = dindex;
  A.obs_point = dindex + M;
  A.point_start = dindex + 2 * size_t(M);
  A.camera_start = A.point_start + P + 1;
  A.camera_obs = A.camera_start + C + 1;
  A.active = A.camera_obs + M;
  A.Hcp = D(o_hcp);
  A.Hcc = D(o_hcc);
  A.Hpp = D(o_hpp);
  A.gc = D(o_gc);
  A.gp = D(o_gp);
  A.Vinv = D(o_vinv);
  A.bp = D(o_bp);
  A.lp = D(o_lp);
  A.yp = D(o_yp);
  A.U = D(o_U);
  A.Minv = D(o_minv);
  A.bc = D(o_bc);
  double* vec = D(o_vec);
  A.x = vec;
  A.r = vec + 6 * size_t(C);
  A.p = vec + 12 * size_t(C);
  A.z = vec + 18 * size_t(C);
  A.Sp = vec + 24 * size_t(C);
  A.cot = D(o_cot);
  A.ybar = D(o_ybar);
  A.state = D(o_state);
  A.tposes = D(o_tposes);
  A.tpoints = D(o_tpoints);
  A.task_obs = reinterpret_cast<const uint32_t*>(a + o_tobs);
  A.part = D(o_part);
  A.mu = 0;
  tba::SchurParams sq{};
  tba::PcgSystem ps{};
  if (schur) {
    Q.bind(d->schur, sq, ps);
    sq.M = M;
    sq.obs_camera = A.obs_camera;
    sq.obs_point = A.obs_point;
    sq.point_start = A.point_start;
    sq.camera_obs = A.camera_obs;
    sq.active = A.active;
    sq.chunk_cam = reinterpret_cast<const uint32_t*>(a + o_ccam);
    sq.chunk_beg = reinterpret_cast<const uint32_t*>(a + o_cbeg);
    sq.cam_chunk = reinterpret_cast<const uint32_t*>(a + o_cfirst);
    sq.A = A.Hcp;
    A.schur = 1;
    A.root = D(o_root);
    A.S = sq.S;
    A.row_ptr = sq.row_ptr;
    A.col = sq.col;
    A.prod_blocks = 0;
    ps.Minv = A.Minv;
    ps.x = A.x;
    ps.r = A.r;
    ps.z = A.z;
    ps.p = A.p;
    ps.state = A.state;
    ps.active = tba::A_ACTIVE;
    ps.failed = tba::A_FAILED;
    ps.converged = ps.inner_r0 = ps.all_steps = -1;
    ps.rho = tba::A_RHO;
    ps.r0 = tba::A_R0;
    ps.r2 = tba::A_R2;
    ps.steps = tba::A_STEPS;
    ps.wait = tba::A_WAIT;
    ps.tol = A.tol;
    ps.alpha_limit = 1e30;
    ps.polls = d->pcg_polls();
  }

  cudaStream_t s = d->stream;
  cudaEvent_t e0 = event(d, 0), e1 = event(d, 1);
  auto up = [&](void* dst, const void* src, size_t bytes) {
    if (bytes) CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
  };
  CUDA_TRY(cudaEventRecord(e0, s));
  up(A.poses, scene, 12 * sizeof(double) * C);
  up(A.points, scene + 12 * size_t(C), 3 * sizeof(double) * P);
  up(const_cast<double*>(A.cams), scene + 12 * size_t(C) + 3 * size_t(P), 6 * sizeof(double) * C);
  up(const_cast<double*>(A.pixels), scene + 18 * size_t(C) + 3 * size_t(P), 2 * sizeof(double) * M);
  up(dindex, index, sizeof(uint32_t) * (3 * size_t(M) + P + 2 * size_t(C) + 2));
  up(const_cast<uint32_t*>(A.task_obs), task_obs.data(), sizeof(uint32_t) * task_obs.size());
  // Before any kernel follows the arrays (scratch: the place of the pixels' cotangent).
  if (checks)
    device_checks(d, *checks, C, P, M, dindex, {A.poses, A.points, A.cams, A.pixels}, reinterpret_cast<uint32_t*>(A.ybar),
                  reinterpret_cast<unsigned long long*>(A.ybar + M));
  uint32_t launches = 0;
  if (schur) {
    up(const_cast<uint32_t*>(sq.chunk_cam), chunks.cam.data(), sizeof(uint32_t) * chunks.cam.size());
    up(const_cast<uint32_t*>(sq.chunk_beg), chunks.beg.data(), sizeof(uint32_t) * chunks.beg.size());
    up(const_cast<uint32_t*>(sq.cam_chunk), chunks.cam_first.data(), sizeof(uint32_t) * chunks.cam_first.size());
    launches += tba::schur_launch_structure(sq, s);
    launches += tba::pcg_launch_plan(ps, Q.grid, s);
  }
  launches += tba::adj_launch_init(A, s);
  CUDA_TRY(cudaGetLastError());

  auto read_state = [&]() {
    CUDA_TRY(cudaMemcpyAsync(d->pinned, A.state, tba::A_WORDS * sizeof(double), cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaStreamSynchronize(s));
    if (d->pinned[tba::A_WAIT] != 0) throw Fail{TBA_ERROR_CUDA, "GPU BA adjoint: a wait between the PCG's blocks ran out"};
  };
  uint32_t cg_total = 0, failed = 0, point_failures = 0;
  const bool time_products = (vc->flags & TBA_VJP_FLAG_TIME_PRODUCTS) != 0;
  double product_ms = 0;
  uint32_t product_launches = 0;
  double last_residual = 0, gnorm_initial = -1, gnorm = 0;
  // One linear solve (H + gauge term) z = rhs by Schur complement and PCG; z lands in x (cameras)
  // and lp (points).  The assembly also measures |F|^2 at the current point.
  auto linear_solve = [&](uint32_t mode, bool cotangent_ready) {
    A.rhs_mode = mode;
    if (!cotangent_ready) launches += tba::adj_launch_reset(A, s);
    launches += tba::adj_launch_assemble(A, s);
    if (schur) launches += tba::schur_launch_values(sq, s);
    launches += tba::adj_launch_pcg_init(A, s);
    CUDA_TRY(cudaGetLastError());
    uint32_t done = 0;
    const bool timed = time_products && (A.prod_blocks || schur);
    // One persistent launch where the system spreads over several blocks.  A system of one block keeps its
    // steps as launches of the graph loop only because the report's kernel_launches is held to count three a
    // PCG step there (tests/test_adjoint.py); one persistent block is the faster form: whole calls at 8, 12, 18
    // and 26 cameras 0.40, 0.41, 0.50 and 0.61 ms against 0.63, 0.71, 0.91 and 1.18.
    const bool persistent = schur && Q.grid > 1 && !timed;
    if (persistent) {
      CUDA_TRY(tba::launch_pcg(ps, vc->max_cg, Q.grid, s));
      launches++;
      done = vc->max_cg;
    }
    const bool on_device = !persistent && !timed && vc->max_cg > 0 && !d->host_pcg_only &&
                           device_loop_ready(d, d->adj_loop, build_adjoint_loop(d->adj_loop, A, s));
    if (on_device) {
      // One launch of the device-side PCG loop, which stops on the device.
      launches += tba::adj_launch_loop_begin(A, vc->max_cg, s);
      CUDA_TRY(cudaGraphLaunch(d->adj_loop.exec, s));
      done = vc->max_cg;
    }
    while (done < vc->max_cg) {
      const uint32_t k = std::min<uint32_t>(16, vc->max_cg - done);
      for (uint32_t j = 0; j < k; j++)
        launches += timed ? tba::adj_launch_pcg_step(A, s, event(d, 8 + 2 * j), event(d, 9 + 2 * j))
                          : tba::adj_launch_pcg_step(A, s);
      CUDA_TRY(cudaGetLastError());
      done += k;
      read_state();
      if (timed) {
        // The chunk's products that ran PCG steps (later launches of a chunk are guarded no-ops).
        const uint32_t steps = uint32_t(d->pinned[tba::A_STEPS]);
        for (uint32_t j = 0; j < k && done - k + j < steps; j++) {
          float ms = 0;
          CUDA_TRY(cudaEventElapsedTime(&ms, event(d, 8 + 2 * j), event(d, 9 + 2 * j)));
          product_ms += ms;
          product_launches++;
        }
      }
      if (d->pinned[tba::A_ACTIVE] == 0) break;
    }
    read_state();
    if (on_device) launches += uint32_t(d->pinned[tba::A_LOOP_ITERS]) * d->adj_loop.body_kernels;
    const double* st = d->pinned;
    cg_total += uint32_t(st[tba::A_STEPS]);
    last_residual = st[tba::A_R0] > 0 ? std::sqrt(st[tba::A_R2] / st[tba::A_R0]) : 0;
    gnorm = std::sqrt(st[tba::A_GNORM]);
    if (gnorm_initial < 0) gnorm_initial = gnorm;
    const bool converged = st[tba::A_R2] <= vc->cg_tolerance * vc->cg_tolerance * st[tba::A_R0] || st[tba::A_R0] == 0;
    if (st[tba::A_POINT_SINGULAR] != 0) failed |= 1;
    point_failures = uint32_t(st[tba::A_POINT_FAILED]);
    if (st[tba::A_CAMERA_FAILED] != 0) failed |= 2;
    if (st[tba::A_FAILED] != 0) failed |= 4;
    if (!converged) failed |= 8;
    launches += tba::adj_launch_back_substitute(A, s);
    CUDA_TRY(cudaGetLastError());
    return st[tba::A_INVALID];
  };
  double invalid = 0;
  // Newton steps on H + mu G (G the IRLS Gauss-Newton matrix): mu shrinks tenfold after a step the
  // robust cost accepts and reaches 0 (exact Newton) below 1e-6, and grows tenfold after a rejected
  // one.  Candidates within a relative 1e-14 of the current cost count as accepted.
  if (vc->newton_steps > 0) {
    launches += tba::adj_launch_cost(A, s);
    read_state();
  }
  double cost = d->pinned[tba::A_COST], mu = 1e-2;
  uint32_t accepted = 0;
  for (uint32_t k = 0; k < vc->newton_steps; k++) {
    A.mu = mu;
    invalid = linear_solve(0, false);
    launches += tba::adj_launch_newton_candidate(A, s);
    CUDA_TRY(cudaGetLastError());
    read_state();
    const double cand = d->pinned[tba::A_COST];
    const bool solved = (failed & 5) == 0;
    failed &= ~uint32_t(13);  // a damped solve that failed is retried with more damping
    if (solved && cand <= cost * (1 + 1e-14)) {
      launches += tba::adj_launch_newton_commit(A, s);
      CUDA_TRY(cudaGetLastError());
      cost = cand;
      accepted++;
      mu = mu < 1e-6 ? 0.0 : mu / 10;
    } else {
      mu = std::max(1e-6, mu * 10);
    }
  }
  A.mu = 0;
  if (cotangent) {
    double* gcot = D(o_gcot);
    up(gcot, cotangent, sizeof(double) * (12 * size_t(C) + 3 * size_t(P)));
    launches += tba::adj_launch_reset(A, s);
    launches += tba::adj_launch_cotangent(A, gcot, s);
    CUDA_TRY(cudaGetLastError());
    invalid = linear_solve(1, true);
    launches += tba::adj_launch_vjp(A, s);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaMemcpyAsync(pixels_bar, A.ybar, 2 * sizeof(double) * M, cudaMemcpyDeviceToHost, s));
    read_state();
    if (intrinsics_bar) {
      intrinsics_bar[0] = d->pinned[tba::A_SBAR];
      intrinsics_bar[1] = d->pinned[tba::A_KBAR];
    }
  } else if (vc->newton_steps > 0) {
    // The gradient at the final point.
    launches += tba::adj_launch_reset(A, s);
    A.rhs_mode = 0;
    launches += tba::adj_launch_assemble(A, s);
    read_state();
    gnorm = std::sqrt(d->pinned[tba::A_GNORM]);
    invalid = d->pinned[tba::A_INVALID];
  }
  if (solution) {
    CUDA_TRY(cudaMemcpyAsync(solution, A.poses, 12 * sizeof(double) * C, cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaMemcpyAsync(solution + 12 * size_t(C), A.points, 3 * sizeof(double) * P, cudaMemcpyDeviceToHost, s));
  }
  CUDA_TRY(cudaEventRecord(e1, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  if (report) {
    std::memset(report, 0, sizeof *report);
    float ms = 0;
    CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
    report->solve_ms = ms;
    report->gradient_norm_initial = gnorm_initial < 0 ? gnorm : gnorm_initial;
    report->gradient_norm_final = gnorm;
    report->adjoint_residual = cotangent ? last_residual : 0;
    report->cg_iterations = cg_total;
    report->newton_steps = accepted;
    report->failed = failed;
    report->invalid = uint32_t(invalid);
    report->point_failures = point_failures;
    report->product_ms = product_ms;
    report->product_launches = product_launches;
    report->product_blocks = A.prod_blocks;
    report->kernel_launches = launches;
    report->wall_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - wall0).count();
  }
}

// ---- observation evaluation ------------------------------------------------------------------------

// (`check`: false is returned, with nothing evaluated, when the device finds the arrays out of order.)
bool evaluate_observations(tba_device* d, const tba_observation_control* oc, const double* cameras,
                           const double* points, const double* pixels, const uint32_t* indices,
                           const uint32_t* offsets, uint32_t* flags, double* summary, tba_observation_report* report,
                           bool check) {
  const auto wall0 = std::chrono::steady_clock::now();
  const uint32_t C = oc->cameras, P = oc->points, M = oc->observations;
  const bool guarded = oc->max_relative_depth_std > 0;
  Layout L;
  const size_t o_cam = L.take<double>(18 * size_t(C)), o_pts = L.take<double>(3 * size_t(P)),
               o_pix = L.take<double>(2 * size_t(M)), o_idx = L.take<uint32_t>(2 * size_t(M)),
               o_off = L.take<uint32_t>(guarded ? size_t(P) + 1 : 0),
               o_flags = L.take<uint32_t>(size_t(M) + (guarded ? P : 0)), o_err = L.take<double>(M),
               o_part = L.take<double>(2 * ((size_t(M) + 63) / 64)), o_sum = L.take<double>(2),
               o_tasks = L.take<uint32_t>(guarded ? size_t(P) + 1 : 0);
  if (d->capacity < L.bytes) {
    if (d->arena) CUDA_TRY(cudaFree(d->arena));
    d->arena = nullptr;
    d->capacity = 0;
    const size_t free_bytes = free_memory(d, L.bytes);
    if (L.bytes > free_bytes)
      throw Fail{TBA_ERROR_BUDGET, "GPU observation evaluation exceeds budget"};
    CUDA_TRY(cudaMalloc(&d->arena, L.bytes));
    d->capacity = L.bytes;
  }
  char* a = d->arena;
  tba::ObsParams p{};
  p.C = C;
  p.P = P;
  p.M = M;
  p.guarded = guarded ? 1 : 0;
  p.max_error = oc->max_error_px;
  p.max_relative_depth = oc->max_relative_depth_std;
  p.noise = oc->pixel_noise_std_px;
  p.cameras = reinterpret_cast<double*>(a + o_cam);
  p.points = reinterpret_cast<double*>(a + o_pts);
  p.pixels = reinterpret_cast<double*>(a + o_pix);
  p.indices = reinterpret_cast<uint32_t*>(a + o_idx);
  p.offsets = guarded ? reinterpret_cast<uint32_t*>(a + o_off) : nullptr;
  p.flags = reinterpret_cast<uint32_t*>(a + o_flags);
  p.errors = reinterpret_cast<double*>(a + o_err);
  p.partials = reinterpret_cast<double*>(a + o_part);
  p.summary = reinterpret_cast<double*>(a + o_sum);
  cudaStream_t s = d->stream;
  cudaEvent_t e0 = event(d, 0), e1 = event(d, 1), e2 = event(d, 2), e3 = event(d, 3);
  uint64_t h2d = 0;
  auto up = [&](size_t off, const void* src, size_t bytes) {
    if (bytes) CUDA_TRY(cudaMemcpyAsync(a + off, src, bytes, cudaMemcpyHostToDevice, s));
    h2d += bytes;
  };
  CUDA_TRY(cudaEventRecord(e0, s));
  up(o_cam, cameras, 18 * sizeof(double) * C);
  up(o_pts, points, 3 * sizeof(double) * P);
  up(o_pix, pixels, 2 * sizeof(double) * M);
  up(o_idx, indices, 2 * sizeof(uint32_t) * M);
  if (guarded) {
    up(o_off, offsets, sizeof(uint32_t) * (size_t(P) + 1));
    // Warp tasks of whole tracks, built while the copies above run.
    const std::vector<uint32_t> tasks = build_tasks(offsets, P);
    p.tasks = reinterpret_cast<uint32_t*>(a + o_tasks);
    p.ntasks = uint32_t(tasks.size() - 1);
    up(o_tasks, tasks.data(), sizeof(uint32_t) * tasks.size());
  }
  CUDA_TRY(cudaEventRecord(e1, s));
  if (check) {
    // Whether the arrays are in order, before any kernel follows their indices.
    tba::ObservationChecks k{};
    k.C = C;
    k.P = P;
    k.M = M;
    k.indices = p.indices;
    k.offsets = p.offsets;
    k.values[0] = p.cameras;
    k.values[1] = p.points;
    k.values[2] = p.pixels;
    k.counts[0] = 18 * uint64_t(C);
    k.counts[1] = 3 * uint64_t(P);
    k.counts[2] = 2 * uint64_t(M);
    k.bad = reinterpret_cast<uint32_t*>(p.summary);  // (written by the evaluation)
    CUDA_TRY(cudaMemsetAsync(k.bad, 0, sizeof(uint32_t), s));
    tba::launch_check_observations(k, d->sms, s);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaMemcpyAsync(d->pinned, k.bad, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaStreamSynchronize(s));
    if (*reinterpret_cast<const uint32_t*>(d->pinned) != 0) return false;
    CUDA_TRY(cudaEventRecord(e1, s));
  }
  tba::launch_observations(p, s);
  CUDA_TRY(cudaGetLastError());
  CUDA_TRY(cudaEventRecord(e2, s));
  const size_t nflags = size_t(M) + (guarded ? P : 0);
  if (nflags) CUDA_TRY(cudaMemcpyAsync(flags, p.flags, nflags * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaMemcpyAsync(summary, p.summary, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaEventRecord(e3, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  if (report) {
    std::memset(report, 0, sizeof *report);
    float ms = 0;
    CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
    report->upload_ms = ms;
    CUDA_TRY(cudaEventElapsedTime(&ms, e1, e2));
    report->evaluate_ms = ms;
    CUDA_TRY(cudaEventElapsedTime(&ms, e2, e3));
    report->download_ms = ms;
    report->h2d_bytes = h2d;
    report->d2h_bytes = nflags * sizeof(uint32_t) + 2 * sizeof(double);
    report->kernel_launches = (guarded ? (p.ntasks ? 1u : 0u) : (M ? 1u : 0u)) + (M ? 1u : 0u) + 1u + (check ? 1u : 0u);
    report->wall_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - wall0).count();
  }
  return true;
}

}  // namespace

extern "C" {

size_t tba_scene_size(const tba_control* c) {
  return c ? 18 * size_t(c->cameras) + 3 * size_t(c->points) + 2 * size_t(c->observations) : 0;
}
size_t tba_index_size(const tba_control* c) {
  return c ? 3 * size_t(c->observations) + c->points + 2 * size_t(c->cameras) + 2 : 0;
}
size_t tba_output_size(const tba_control* c) {
  return c ? 12 * size_t(c->cameras) + 3 * size_t(c->points) + 26 + (c->shared_focal ? 1 : 0) : 0;
}

tba_status tba_device_open(int ordinal, tba_device** out) {
  if (!out) return TBA_ERROR_ARGUMENT;
  *out = nullptr;
  int count = 0;
  cudaError_t e = cudaGetDeviceCount(&count);
  if (e != cudaSuccess || count == 0) {
    g_open_error = std::string("no CUDA device: ") + cudaGetErrorString(e);
    return TBA_ERROR_INTERNAL;
  }
  if (ordinal < 0 || ordinal >= count) {
    g_open_error = "CUDA device ordinal out of range";
    return TBA_ERROR_ARGUMENT;
  }
  tba_device* d = new tba_device();
  d->ordinal = ordinal;
  try {
    CUDA_TRY(cudaSetDevice(ordinal));
    cudaDeviceProp prop;
    CUDA_TRY(cudaGetDeviceProperties(&prop, ordinal));
    if (prop.major < 10) throw Fail{TBA_ERROR_INTERNAL, "libtba.so is built for sm_100a (B200); device is sm_" +
                                                            std::to_string(prop.major) + std::to_string(prop.minor)};
    d->sms = prop.multiProcessorCount;
    CUDA_TRY(cudaStreamCreateWithFlags(&d->stream, cudaStreamNonBlocking));
    CUDA_TRY(cudaStreamCreateWithFlags(&d->down, cudaStreamNonBlocking));
    CUDA_TRY(cudaMallocHost(&d->pinned, 128 * sizeof(double)));
    CUDA_TRY(tba::configure_kernels());
    CUDA_TRY(tba::pcg_configure());
    CUDA_TRY(tba::adj_configure());
    CUDA_TRY(tba::batch_configure());
  } catch (const Fail& f) {
    g_open_error = f.message;
    tba_device_close(d);
    return f.status;
  }
  *out = d;
  return TBA_OK;
}

void tba_device_close(tba_device* d) {
  if (!d) return;
  cudaSetDevice(d->ordinal);
  if (d->stream) cudaStreamSynchronize(d->stream);
  if (d->down) cudaStreamSynchronize(d->down);
  for (cudaEvent_t e : d->events) cudaEventDestroy(e);
  if (d->batch_graph) cudaGraphExecDestroy(d->batch_graph);
  if (d->window_graph) cudaGraphExecDestroy(d->window_graph);
  for (PcgLoop& loop : d->pcg_loops) loop.release();
  d->adj_loop.release();
  if (d->batch_arena) cudaFree(d->batch_arena);
  if (d->arena) cudaFree(d->arena);
  if (d->schur) cudaFree(d->schur);
  if (d->pinned) cudaFreeHost(d->pinned);
  if (d->stream) cudaStreamDestroy(d->stream);
  if (d->down) cudaStreamDestroy(d->down);
  delete d;
}

const char* tba_last_error(const tba_device* d) { return d ? d->error.c_str() : g_open_error.c_str(); }

tba_status tba_bundle_adjust(tba_device* d, const tba_control* control, const double* scene, size_t scene_len,
                             const uint32_t* index, size_t index_len, double* output, size_t output_len,
                             tba_report* report) {
  if (!d) return TBA_ERROR_ARGUMENT;
  std::lock_guard<std::mutex> lock(d->mu);
  d->error.clear();
  try {
    check_control(control);
    if (!scene || !index || !output) argument("Invalid GPU BA arrays: null pointer");
    if (scene_len != tba_scene_size(control)) argument("Invalid GPU BA scene array length");
    if (index_len != tba_index_size(control)) argument("Invalid GPU BA index array length");
    if (output_len < tba_output_size(control)) argument("Invalid GPU BA output array length");
    if (uint64_t(3) * control->observations + control->points + 2ull * control->cameras + 2 > 0xffffffffull)
      argument("GPU BA scene dimensions exceed integer index bounds");
    // The O(C) checks here, the O(M) ones on the device after the upload (before any solver kernel).
    const auto t0 = std::chrono::steady_clock::now();
    const HostChecks hc = host_checks(control, index, scene);
    double check_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    CUDA_TRY(cudaSetDevice(d->ordinal));
    SolveIO io;
    io.checks = &hc;
    io.check_ms = &check_ms;
    solve(d, control, scene, index, output, report, io);
    if (report) report->check_ms = check_ms;
  } catch (const Fail& f) {
    d->error = f.message;
    return f.status;
  } catch (const std::exception& e) {
    d->error = e.what();
    return TBA_ERROR_INTERNAL;
  }
  return TBA_OK;
}

uint32_t tba_batch_max_cameras(void) { return tba::batch_max_cameras(); }
uint32_t tba_batch_shapes(void) { return uint32_t(tba::kBatchShapes) + 1; }

tba_status tba_batch_shape(uint32_t k, uint32_t* threads, uint32_t* min_blocks) {
  if (k > uint32_t(tba::kBatchGridShape)) return TBA_ERROR_ARGUMENT;
  const tba::BatchShape s = k == uint32_t(tba::kBatchGridShape) ? tba::BatchShape{tba::kBatchGridThreads, 2} : tba::batch_shape(int(k));
  if (threads) *threads = uint32_t(s.threads);
  if (min_blocks) *min_blocks = uint32_t(s.min_blocks);
  return TBA_OK;
}

tba_status tba_batch_adjust(tba_device* d, const tba_batch_control* control, const tba_batch_problem* problems,
                            uint32_t count, const double* scene, size_t scene_len, const uint32_t* index,
                            size_t index_len, double* output, size_t output_len, tba_batch_report* report) {
  if (!d) return TBA_ERROR_ARGUMENT;
  std::lock_guard<std::mutex> lock(d->mu);
  d->error.clear();
  try {
    if (!control) argument("Invalid GPU BA batch: no control block");
    if (count == 0 || !problems) argument("Invalid GPU BA batch: no problems");
    if (!scene || !index || !output) argument("Invalid GPU BA arrays: null pointer");
    CUDA_TRY(cudaSetDevice(d->ordinal));
    solve_batch(d, control, problems, count, scene, scene_len, index, index_len, output, output_len, report);
  } catch (const Fail& f) {
    d->error = f.message;
    return f.status;
  } catch (const std::exception& e) {
    d->error = e.what();
    return TBA_ERROR_INTERNAL;
  }
  return TBA_OK;
}

tba_status tba_bundle_vjp(tba_device* d, const tba_vjp_control* vc, const double* scene, size_t scene_len,
                          const uint32_t* index, size_t index_len, const double* cotangent, size_t cotangent_len,
                          double* pixels_bar, size_t pixels_bar_len, double* intrinsics_bar, double* solution,
                          size_t solution_len, tba_vjp_report* report) {
  if (!d) return TBA_ERROR_ARGUMENT;
  std::lock_guard<std::mutex> lock(d->mu);
  d->error.clear();
  try {
    if (!vc) argument("Invalid GPU BA adjoint: no control block");
    tba_control c{};
    c.cameras = vc->cameras;
    c.points = vc->points;
    c.observations = vc->observations;
    c.anchor = vc->anchor;
    c.scale_view = vc->scale_view;
    c.iterations = 0;
    c.max_cg = 1;
    c.huber = vc->huber;
    c.cg_tolerance = 1e-6;
    c.stall_tolerance = 1e-9;
    check_control(&c);
    if (vc->newton_steps > 50 || vc->max_cg < 1 || vc->max_cg > 100000 || (vc->flags & ~TBA_VJP_FLAG_TIME_PRODUCTS) != 0 ||
        !(std::isfinite(vc->cg_tolerance) && vc->cg_tolerance >= 1e-15 && vc->cg_tolerance <= 1e-2))
      argument("Invalid GPU BA adjoint options");
    if (!scene || !index) argument("Invalid GPU BA arrays: null pointer");
    if (scene_len != tba_scene_size(&c)) argument("Invalid GPU BA scene array length");
    if (index_len != tba_index_size(&c)) argument("Invalid GPU BA index array length");
    const size_t n_theta = 12 * size_t(c.cameras) + 3 * size_t(c.points);
    if (cotangent && (cotangent_len != n_theta || !pixels_bar || pixels_bar_len < 2 * size_t(c.observations)))
      argument("Invalid GPU BA adjoint arrays: the cotangent needs 12C + 3P values and pixels_bar 2M");
    if (solution && solution_len < n_theta) argument("Invalid GPU BA adjoint arrays: solution needs 12C + 3P values");
    if (cotangent)
      for (size_t i = 0; i < n_theta; i++)
        if (!std::isfinite(cotangent[i])) argument("Invalid GPU BA adjoint: the cotangent is not finite");
    if (uint64_t(3) * c.observations + c.points + 2ull * c.cameras + 2 > 0xffffffffull)
      argument("GPU BA scene dimensions exceed integer index bounds");
    const bool on_device = c.observations >= kDeviceCheckMin;
    auto host_check = [&] {
      check_index(&c, index);
      check_scene(&c, scene, scene_len);
    };
    if (!on_device) host_check();
    const HostChecks checks = on_device ? host_checks(&c, index, scene) : HostChecks{};
    try {
      CUDA_TRY(cudaSetDevice(d->ordinal));
      solve_vjp(d, vc, on_device ? &checks : nullptr, scene, index, cotangent, pixels_bar, intrinsics_bar, solution, report);
    } catch (const Fail& f) {
      if (on_device && f.status == TBA_ERROR_BUDGET) host_check();  // arrays out of order are reported first
      throw;
    }
  } catch (const Fail& f) {
    d->error = f.message;
    return f.status;
  } catch (const std::exception& e) {
    d->error = e.what();
    return TBA_ERROR_INTERNAL;
  }
  return TBA_OK;
}

tba_status tba_evaluate_observations(tba_device* d, const tba_observation_control* oc, const double* cameras,
                                     size_t cameras_len, const double* points, size_t points_len, const double* pixels,
                                     size_t pixels_len, const uint32_t* indices, size_t indices_len,
                                     const uint32_t* offsets, size_t offsets_len, uint32_t* flags, size_t flags_len,
                                     double* summary, tba_observation_report* report) {
  if (!d) return TBA_ERROR_ARGUMENT;
  std::lock_guard<std::mutex> lock(d->mu);
  d->error.clear();
  try {
    if (!oc || !summary) argument("Invalid GPU observation request");
    const uint64_t C = oc->cameras, P = oc->points, M = oc->observations;
    const bool guarded = oc->max_relative_depth_std > 0;
    if (!(std::isfinite(oc->max_error_px) && oc->max_error_px >= 1e-12 && oc->max_error_px <= 1e6) ||
        !(std::isfinite(oc->max_relative_depth_std) && oc->max_relative_depth_std >= 0 &&
          oc->max_relative_depth_std <= 1e9) ||
        !(std::isfinite(oc->pixel_noise_std_px) && oc->pixel_noise_std_px > 0 && oc->pixel_noise_std_px <= 1e9))
      argument("Invalid GPU observation threshold");
    if (2 * M + P + 1 > 0xffffffffull || 18 * C > 0xffffffffull || 8 * P > 0xffffffffull)
      argument("GPU observation evaluation exceeds budget");
    if ((C && !cameras) || (P && !points) || (M && (!pixels || !indices)) || ((M || guarded) && !flags))
      argument("Invalid GPU observation arrays: null pointer");
    if (cameras_len < 18 * C || points_len < 3 * P || pixels_len < 2 * M || indices_len < 2 * M ||
        flags_len < M + (guarded ? P : 0))
      argument("Invalid GPU observation arrays: lengths");
    // The O(M) checks run on the device after the upload; the host makes them where the device finds the
    // arrays out of order, for the message a serial scan meets first, and on small calls.
    auto host_check = [&] {
      FirstFailure ff;
      parallel_ranges(M, 1u << 18, [&](uint64_t b, uint64_t e, unsigned) {
        for (uint64_t i = b; i < e; i++)
          if (indices[2 * i] >= C || indices[2 * i + 1] >= P)
            return ff.record(i, "Invalid GPU observation indices: a camera or point out of range");
      });
      ff.raise();
      if (guarded) {
        if (!offsets || offsets_len < P + 1) argument("Invalid GPU observation arrays: track offsets");
        if (offsets[0] != 0 || offsets[P] != M) argument("Invalid GPU observation arrays: track offsets");
        FirstFailure tf;
        parallel_ranges(P, 1u << 16, [&](uint64_t b, uint64_t e, unsigned) {
          for (uint64_t h = b; h < e; h++) {
            if (offsets[h + 1] < offsets[h] || offsets[h + 1] > M)
              return tf.record(h, "Invalid GPU observation arrays: track offsets");
            for (uint64_t i = offsets[h]; i < offsets[h + 1]; i++)
              if (indices[2 * i + 1] != h) return tf.record(h, "Invalid GPU observation arrays: track offsets");
          }
        });
        tf.raise();
      }
      FirstFailure bf;
      auto bounded = [&](const double* v, uint64_t n, uint64_t base) {
        parallel_ranges(n, 1u << 18, [&](uint64_t b, uint64_t e, unsigned) {
          for (uint64_t i = b; i < e; i++) {
            const double x = v[i];
            if (!std::isfinite(x) || std::fabs(x) > 1e9 || (x != 0 && std::fabs(x) < 1e-30))
              return bf.record(base + i, "Invalid GPU scene coordinate bounds");
          }
        });
      };
      bounded(cameras, 18 * C, 0);
      bounded(points, 3 * P, 18 * C);
      bounded(pixels, 2 * M, 18 * C + 3 * P);
      bf.raise();
    };
    const bool on_device = M >= kDeviceCheckMin && !(guarded && (!offsets || offsets_len < P + 1));
    if (!on_device) host_check();
    if (on_device && guarded && (offsets[0] != 0 || offsets[P] != M)) host_check();
    try {
      CUDA_TRY(cudaSetDevice(d->ordinal));
      if (!evaluate_observations(d, oc, cameras, points, pixels, indices, offsets, flags, summary, report, on_device)) {
        host_check();
        throw Fail{TBA_ERROR_INTERNAL, "GPU observation checks disagree"};
      }
    } catch (const Fail& f) {
      if (on_device && f.status == TBA_ERROR_BUDGET) host_check();  // arrays out of order are reported first
      throw;
    }
  } catch (const Fail& f) {
    d->error = f.message;
    return f.status;
  } catch (const std::exception& e) {
    d->error = e.what();
    return TBA_ERROR_INTERNAL;
  }
  return TBA_OK;
}

tba_status tba_scene_create(tba_device* d, const tba_control* shape, const double* scene, size_t scene_len,
                            const uint32_t* index, size_t index_len, tba_scene** out) {
  if (!d || !out) return TBA_ERROR_ARGUMENT;
  *out = nullptr;
  std::lock_guard<std::mutex> lock(d->mu);
  d->error.clear();
  tba_scene* r = nullptr;
  try {
    check_control(shape);
    if (!scene || !index) argument("Invalid GPU BA arrays: null pointer");
    if (scene_len != tba_scene_size(shape)) argument("Invalid GPU BA scene array length");
    if (index_len != tba_index_size(shape)) argument("Invalid GPU BA index array length");
    if (uint64_t(3) * shape->observations + shape->points + 2ull * shape->cameras + 2 > 0xffffffffull)
      argument("GPU BA scene dimensions exceed integer index bounds");
    check_index(shape, index);
    check_scene(shape, scene, scene_len);
    CUDA_TRY(cudaSetDevice(d->ordinal));
    r = new tba_scene();
    r->device = d;
    r->shape = *shape;
    HostPlan* plan = new HostPlan(make_plan(shape, index, d->sms));
    r->plan = plan;
    plan->tracks = survey(shape->cameras, shape->points, shape->observations, index);
    std::vector<uint32_t> flat;
    for (const std::vector<uint32_t>* v : static_cast<HostPlan*>(r->plan)->sections()) flat.insert(flat.end(), v->begin(), v->end());
    // (an explicit system's buffer that the handle keeps from its last solve makes room for the scene)
    free_memory(d, scene_len * sizeof(double) + (index_len + flat.size()) * sizeof(uint32_t) + 3 * kAllocationGrain);
    CUDA_TRY(cudaMalloc(&r->scene, scene_len * sizeof(double)));
    CUDA_TRY(cudaMalloc(&r->index, index_len * sizeof(uint32_t)));
    CUDA_TRY(cudaMalloc(&r->plan_dev, std::max<size_t>(1, flat.size()) * sizeof(uint32_t)));
    CUDA_TRY(cudaMemcpyAsync(r->scene, scene, scene_len * sizeof(double), cudaMemcpyHostToDevice, d->stream));
    CUDA_TRY(cudaMemcpyAsync(r->index, index, index_len * sizeof(uint32_t), cudaMemcpyHostToDevice, d->stream));
    CUDA_TRY(cudaMemcpyAsync(r->plan_dev, flat.data(), flat.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, d->stream));
    CUDA_TRY(cudaStreamSynchronize(d->stream));
  } catch (const Fail& f) {
    d->error = f.message;
    if (r) {
      if (r->scene) cudaFree(r->scene);
      if (r->index) cudaFree(r->index);
      if (r->plan_dev) cudaFree(r->plan_dev);
      delete static_cast<HostPlan*>(r->plan);
      delete r;
    }
    return f.status;
  }
  *out = r;
  return TBA_OK;
}

void tba_scene_destroy(tba_scene* r) {
  if (!r) return;
  {
    std::lock_guard<std::mutex> lock(r->device->mu);
    cudaSetDevice(r->device->ordinal);
    cudaStreamSynchronize(r->device->stream);
    if (r->scene) cudaFree(r->scene);
    if (r->index) cudaFree(r->index);
    if (r->plan_dev) cudaFree(r->plan_dev);
  }
  delete static_cast<HostPlan*>(r->plan);
  delete r;
}

tba_status tba_scene_adjust(tba_device* d, tba_scene* r, const tba_control* control, double* output,
                            size_t output_len, double* state, size_t state_len, tba_report* report) {
  if (!d || !r) return TBA_ERROR_ARGUMENT;
  std::lock_guard<std::mutex> lock(d->mu);
  d->error.clear();
  try {
    if (r->device != d) argument("Invalid GPU BA resident scene: it belongs to another device handle");
    check_control(control);
    const tba_control& s = r->shape;
    if (control->cameras != s.cameras || control->points != s.points || control->observations != s.observations ||
        control->directional_points != s.directional_points || control->anchor != s.anchor ||
        control->scale_view != s.scale_view)
      argument("Invalid GPU BA resident scene: the control's sizes or gauge differ from the scene's");
    if (output && output_len < tba_output_size(control)) argument("Invalid GPU BA output array length");
    if (state && state_len < size_t(26 + (control->shared_focal ? 1 : 0))) argument("Invalid GPU BA state array length");
    CUDA_TRY(cudaSetDevice(d->ordinal));
    SolveIO io;
    io.device_source = true;
    io.plan = static_cast<const HostPlan*>(r->plan);
    io.plan_dev = r->plan_dev;
    io.writeback = r->scene;
    io.state = state;
    solve(d, control, r->scene, r->index, output, report, io);
    if (report) report->check_ms = 0;
  } catch (const Fail& f) {
    d->error = f.message;
    return f.status;
  } catch (const std::exception& e) {
    d->error = e.what();
    return TBA_ERROR_INTERNAL;
  }
  return TBA_OK;
}

tba_status tba_scene_write(tba_device* d, tba_scene* r, const double* poses, const double* points) {
  if (!d || !r) return TBA_ERROR_ARGUMENT;
  std::lock_guard<std::mutex> lock(d->mu);
  d->error.clear();
  try {
    if (r->device != d) argument("Invalid GPU BA resident scene: it belongs to another device handle");
    const size_t C = r->shape.cameras, P = r->shape.points;
    auto bounded = [](const double* v, size_t n) {
      for (size_t i = 0; i < n; i++) {
        const double x = v[i];
        if (!std::isfinite(x) || std::fabs(x) > 1e9 || (x != 0 && std::fabs(x) < 1e-30)) return false;
      }
      return true;
    };
    if ((poses && !bounded(poses, 12 * C)) || (points && !bounded(points, 3 * P)))
      argument("GPU BA input exceeds supported coordinate bounds");
    CUDA_TRY(cudaSetDevice(d->ordinal));
    if (poses) CUDA_TRY(cudaMemcpyAsync(r->scene, poses, 12 * C * sizeof(double), cudaMemcpyHostToDevice, d->stream));
    if (points)
      CUDA_TRY(cudaMemcpyAsync(r->scene + 12 * C, points, 3 * P * sizeof(double), cudaMemcpyHostToDevice, d->stream));
    CUDA_TRY(cudaStreamSynchronize(d->stream));
  } catch (const Fail& f) {
    d->error = f.message;
    return f.status;
  }
  return TBA_OK;
}

tba_status tba_scene_read(tba_device* d, tba_scene* r, double* poses, double* points) {
  if (!d || !r) return TBA_ERROR_ARGUMENT;
  std::lock_guard<std::mutex> lock(d->mu);
  d->error.clear();
  try {
    if (r->device != d) argument("Invalid GPU BA resident scene: it belongs to another device handle");
    const size_t C = r->shape.cameras, P = r->shape.points;
    CUDA_TRY(cudaSetDevice(d->ordinal));
    if (poses) CUDA_TRY(cudaMemcpyAsync(poses, r->scene, 12 * C * sizeof(double), cudaMemcpyDeviceToHost, d->stream));
    if (points)
      CUDA_TRY(cudaMemcpyAsync(points, r->scene + 12 * C, 3 * P * sizeof(double), cudaMemcpyDeviceToHost, d->stream));
    CUDA_TRY(cudaStreamSynchronize(d->stream));
  } catch (const Fail& f) {
    d->error = f.message;
    return f.status;
  }
  return TBA_OK;
}

tba_status tba_device_set_wait_limit(tba_device* d, uint32_t polls) {
  if (!d) return TBA_ERROR_ARGUMENT;
  std::lock_guard<std::mutex> lock(d->mu);
  d->wait_limit = polls;
  return TBA_OK;
}

// Rows per slice of an inverse-depth call (2,048 tiles of 128 rows; at most 8 slices a call).
constexpr uint32_t kIdSliceRows = 1u << 18;

tba_status tba_linearize_inverse_depth(tba_device* d, uint32_t count, const double* measurements,
                                       size_t measurements_len, double* linearizations, size_t linearizations_len,
                                       tba_observation_report* report) {
  if (!d) return TBA_ERROR_ARGUMENT;
  std::lock_guard<std::mutex> lock(d->mu);
  d->error.clear();
  try {
    if (count && (!measurements || !linearizations)) argument("Invalid inverse-depth arrays: null pointer");
    if (measurements_len < 34ull * count || linearizations_len < 23ull * count)
      argument("Invalid inverse-depth arrays: lengths");
    if (34ull * count > 0xffffffffull) argument("Inverse-depth measurement budget cannot fit the observations");
    // Values are not checked, as the reference kernel's are not: a row whose projection leaves the
    // camera model's domain comes back with a zero flag.
    CUDA_TRY(cudaSetDevice(d->ordinal));
    const auto wall0 = std::chrono::steady_clock::now();
    Layout L;
    const size_t o_in = L.take<double>(34 * size_t(count)), o_out = L.take<double>(23 * size_t(count));
    const size_t o_err = L.take<uint32_t>(1);
    if (d->capacity < L.bytes) {
      if (d->arena) CUDA_TRY(cudaFree(d->arena));
      d->arena = nullptr;
      d->capacity = 0;
      const size_t free_bytes = free_memory(d, L.bytes);
      if (L.bytes > free_bytes) throw Fail{TBA_ERROR_BUDGET, "Inverse-depth measurement budget cannot fit the observations"};
      CUDA_TRY(cudaMalloc(&d->arena, L.bytes));
      d->capacity = L.bytes;
    }
    double* din = reinterpret_cast<double*>(d->arena + o_in);
    double* dout = reinterpret_cast<double*>(d->arena + o_out);
    uint32_t* derr = reinterpret_cast<uint32_t*>(d->arena + o_err);
    uint32_t err = 0;
    cudaStream_t s = d->stream, down = d->down;
    // Slices of whole 128-row tiles (so every slice's rows start 16-byte aligned in both arrays):
    // slice j's upload and kernel run on the main stream, its download on the second stream once
    // its kernel is done, so downloads overlap the next slices' uploads (the link is full duplex)
    // and the call takes about one upload plus one slice's kernel and download.
    const uint32_t slices = count <= kIdSliceRows ? 1u : std::min<uint32_t>(8u, (count + kIdSliceRows - 1) / kIdSliceRows);
    const uint32_t per = slices == 1 ? count : ((count + slices - 1) / slices + 127) / 128 * 128;
    // Events: per slice [upload start, upload end = kernel start, kernel end, download start,
    // download end], then the call's end on the second stream.
    CUDA_TRY(cudaMemsetAsync(derr, 0, sizeof(uint32_t), s));
    uint32_t launched = 0;
    for (uint32_t j = 0, first = 0; first < count; j++, first += per) {
      const uint32_t n = std::min(per, count - first);
      cudaEvent_t ev[5];
      for (int k = 0; k < 5; k++) ev[k] = event(d, 5 * size_t(j) + k);
      CUDA_TRY(cudaEventRecord(ev[0], s));
      CUDA_TRY(cudaMemcpyAsync(din + 34 * size_t(first), measurements + 34 * size_t(first), 34 * sizeof(double) * n,
                               cudaMemcpyHostToDevice, s));
      CUDA_TRY(cudaEventRecord(ev[1], s));
      CUDA_TRY(tba::launch_linearize_inverse_depth(n, din + 34 * size_t(first), dout + 23 * size_t(first), derr,
                                                   d->sms, s, d->wait_limit));
      launched++;
      CUDA_TRY(cudaEventRecord(ev[2], s));
      CUDA_TRY(cudaStreamWaitEvent(down, ev[2], 0));
      CUDA_TRY(cudaEventRecord(ev[3], down));
      CUDA_TRY(cudaMemcpyAsync(linearizations + 23 * size_t(first), dout + 23 * size_t(first),
                               23 * sizeof(double) * n, cudaMemcpyDeviceToHost, down));
      CUDA_TRY(cudaEventRecord(ev[4], down));
    }
    CUDA_TRY(cudaMemcpyAsync(&err, derr, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaStreamSynchronize(s));
    CUDA_TRY(cudaStreamSynchronize(down));
    if (err == 1) throw Fail{TBA_ERROR_CUDA, "Inverse-depth linearization: a tile load did not complete"};
    if (err) throw Fail{TBA_ERROR_CUDA, "Inverse-depth linearization: a tile load did not complete, and the loads "
                                        "in flight after it did not land in time"};
    if (report) {
      std::memset(report, 0, sizeof *report);
      // Sums over the slices (the phases of different slices overlap).
      for (uint32_t j = 0; j < launched; j++) {
        float ms = 0;
        CUDA_TRY(cudaEventElapsedTime(&ms, event(d, 5 * size_t(j)), event(d, 5 * size_t(j) + 1)));
        report->upload_ms += ms;
        CUDA_TRY(cudaEventElapsedTime(&ms, event(d, 5 * size_t(j) + 1), event(d, 5 * size_t(j) + 2)));
        report->evaluate_ms += ms;
        CUDA_TRY(cudaEventElapsedTime(&ms, event(d, 5 * size_t(j) + 3), event(d, 5 * size_t(j) + 4)));
        report->download_ms += ms;
      }
      report->h2d_bytes = 34ull * 8 * count;
      report->d2h_bytes = 23ull * 8 * count;
      report->kernel_launches = launched;
      report->wall_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - wall0).count();
    }
  } catch (const Fail& f) {
    d->error = f.message;
    return f.status;
  }
  return TBA_OK;
}

}  // extern "C"
