// Device code of the GB300 DVS hot path (sm_103a).
//
// Built with -fmad=false: every floating-point expression rounds exactly as
// the reference writes it (and as the oracle computes it on the CPU), so the
// ray directions, Moller-Trumbore results and shadow origins differ from the
// reference only where CUDA's transcendental functions differ from the host C
// library (quotients and roots: device_math.cuh), and the FP64 circuit by the
// last bits of its receptor step (device_circuit.cuh).
//
// Work decomposition
//   * trace_cells: a warp's item is many packets of 32 (pixel, cell) samples --
//     32/CW Morton-adjacent pixels x CW consecutive circuit cells -- over the
//     pixel's sub-rays, several cell groups and pixels.  Items with enough
//     packets walk the 8-wide BVH once for all of them (the beam,
//     device_optics.cuh) and test the leaves it reaches; the others walk it per
//     packet, all lanes together: coherent packets test one child per lane
//     against the packet's ray intervals, leaves are tested per lane, and each
//     lane keeps its own closest hit.  The stack and the lists live in shared memory.
//   * trace_poses: few poses a pixel (frames, initial pose, probes): packets of
//     one or more pixels' sub-rays, items of several pixels through one beam.
//   * circuit: one thread per pixel streams the per-cell radiance of a chunk
//     and integrates the pixel circuit (pixel_model.hpp semantics).
//   * emit_events: warp prefix-sum compaction of the per-pixel event slabs.
//   * event_depth: depth re-trace at each event time, a warp per event (event_sensor.cu:51-59).
#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>
#include <curand_kernel.h>

#include "kernels.h"
#include "device_optics.cuh"
#include "device_circuit.cuh"
#include "trace_item.cuh"

namespace dvsgb {
namespace {

// ---- kernels ------------------------------------------------------------------------
__global__ void hapke_const_kernel(dvs_hapke p, HapkeConst *out) { *out = hapke_const(p); }

__global__ void pose_from_state_kernel(const dvs_optical_state *state, CellPose *out) {
  // A pose used as given (initialize_pixels, event_sensor.cu:22): the
  // quaternion is not renormalized; only the light is normalized.
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const dvs_optical_state s = *state;
  const float3 ln = normalize(ld3(s.light));
  CellPose o;
  o.px = s.position.x; o.py = s.position.y; o.pz = s.position.z; o.intensity = s.intensity;
  o.qx = s.rotation.x; o.qy = s.rotation.y; o.qz = s.rotation.z; o.qw = s.rotation.w;
  o.lx = ln.x; o.ly = ln.y; o.lz = ln.z; o.pad = 0;
  *out = o;
}

__global__ void poses_from_states_kernel(const dvs_optical_state *states, int n, CellPose *out) {
  // pose_from_state_kernel for n states: pose as given, light normalized
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const dvs_optical_state s = states[i];
  const float3 ln = normalize(ld3(s.light));
  CellPose o;
  o.px = s.position.x; o.py = s.position.y; o.pz = s.position.z; o.intensity = s.intensity;
  o.qx = s.rotation.x; o.qy = s.rotation.y; o.qz = s.rotation.z; o.qw = s.rotation.w;
  o.lx = ln.x; o.ly = ln.y; o.lz = ln.z; o.pad = 0;
  out[i] = o;
}

__global__ void cell_poses_kernel(const dvs_optical_interval *ivs, const Cell *cells, int n, CellPose *out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  const Cell cell = cells[c];
  out[c] = pose_at(ivs[cell.interval], (cell.t0 + cell.t1) * .5);
}


template <int kMode, int kRays, int kGeo, bool kBeam>
__global__ void __launch_bounds__(128, kRays == 4   ? DVS_TRACE_QUAD_MIN_BLOCKS
                                       : kRays == 2 ? DVS_TRACE_PAIR_MIN_BLOCKS
                                       : kBeam      ? DVS_TRACE_BEAM_MIN_BLOCKS
                                                    : DVS_TRACE_MIN_BLOCKS)
    trace_cells_kernel(const __grid_constant__ SceneView S, int n_pix, const int32_t *rank_list, const CellPose *poses,
                       int c0, int nc, ItemShape shape, double *radiance, float *depth_out,
                       unsigned long long *counters) {
  __shared__ TraceShared s_warp[kWarpsPerBlock];
  __shared__ Beam s_beam[kBeam ? kWarpsPerBlock : 1];
  const int wib = threadIdx.x >> 5;
  const long long item = (long long)blockIdx.x * kWarpsPerBlock + wib;
  trace_cells_item<kMode, kRays, kGeo, kBeam>(S, n_pix, rank_list, poses, c0, nc, shape, radiance, depth_out, counters, item,
                                       s_warp[wib], s_beam[kBeam ? wib : 0]);
}

template <int kMode, int kGeo>
__global__ void __launch_bounds__(128, 4)
    trace_poses_kernel(const __grid_constant__ SceneView S, int n_pix, const int32_t *rank_list, const CellPose *poses,
                       int c0, int nc, PoseShape shape, double *radiance, float *depth_out,
                       unsigned long long *counters) {
  __shared__ PoseShared s_warp[kWarpsPerBlock];
  const int wib = threadIdx.x >> 5;
  const long long item = (long long)blockIdx.x * kWarpsPerBlock + wib;
  const long long first = item / nc * shape.pixels;
  if (first >= n_pix) return;  // warp-uniform
  const int cell = (int)(item % nc);
  const CellPose pose = poses[c0 + cell];
  trace_pose_item<kMode, kGeo>(S, n_pix, rank_list, pose, cell, shape, radiance, depth_out, counters, (int)first,
                               s_warp[wib]);
}

template <class Rng>
__global__ void init_pixels_kernel(int n, const int32_t *pixel_of_rank, const double *radiance, PixelParams p,
                                   PhotoParams photo, double stddev, double minimum, unsigned seed, CircuitState st,
                                   int32_t *error) {
  // initialize_pixels (event_sensor.cu:18-28); Rng = XORWOW (the reference's
  // generator) or, in precision mode, the head of the pixel's Philox stream
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int pixel = pixel_of_rank[k];
  Rng rng;
  curand_init(seed, pixel, 0, &rng);
  const double rad = radiance[k];
  if (!isfinite(rad)) {
    atomicOr(error, kErrOptical);
    if constexpr (std::is_same<Rng, curandStateXORWOW_t>::value) st.rng[k] = rng;
    return;
  }
  const double u = log(fmax(1e-30, rad * photo.electrons_per_radiance + photo.dark_electrons));
  st.receptor_log[k] = u;
  st.receptor[k] = exp(u);
  st.reference_log[k] = u;
  st.refractory_until[k] = -1;
  st.threshold_pos[k] = fmax(minimum, p.threshold_pos + stddev * curand_normal_double(&rng));
  st.threshold_neg[k] = fmax(minimum, p.threshold_neg + stddev * curand_normal_double(&rng));
  st.reset_pending[k] = 0;
  if constexpr (std::is_same<Rng, curandStateXORWOW_t>::value) st.rng[k] = rng;
}

// The photon counts of a float radiance chunk, in place, as rates: the draw of circuit_rank's Philox cells, a thread per
// pixel-cell.
__global__ void __launch_bounds__(128) philox_draws_kernel(int n, const Cell *cells, int c0, int nc,
                                                           const int32_t *pixel_of_rank, PhotoParams photo,
                                                           float *chunk) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)n * nc) return;
  const int c = (int)(i / n), r = (int)(i - (long long)c * n);
  const float rad = chunk[i];
  const Cell cell = cells[c0 + c];
  // a radiance that is not finite stays for the circuit to report; a cell of no length draws nothing (its rate would be
  // 0 / 0, which the circuit would report too), and the circuit passes over it
  if (!isfinite(rad) || !(cell.dt > 0.0f)) return;
  chunk[i] = philox_rate(photo, rad * (float)photo.electrons_per_radiance + (float)photo.dark_electrons,
                         pixel_of_rank[r], cell);
}

template <bool kF32, bool kPhilox>
__global__ void __launch_bounds__(128) circuit_kernel(int n, const int32_t *rank_list, const Cell *cells, int c0,
                                                      int nc, const double *radiance, PixelParams p,
                                                      PhotoParams photo, int max_events, CircuitState st,
                                                      int32_t *ev_count, double *slab_t, int8_t *slab_p,
                                                      int32_t *error, unsigned long long *counters) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  circuit_rank<kF32, kPhilox>(r, n, rank_list, cells, c0, nc, radiance, p, photo, max_events, st, ev_count, slab_t,
                              slab_p, error, counters);
}

__global__ void emit_events_kernel(int n, const int32_t *pixel_of_rank, int width, int max_events,
                                   const int32_t *ev_count, const double *slab_t, const int8_t *slab_p,
                                   DevEvent *out, int32_t *out_count) {
  // warp ballot/prefix-sum compaction; one atomic per warp
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const int cnt = (k < n && ev_count[k] > 0) ? ev_count[k] : 0;
  int incl = cnt;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    int v = __shfl_up_sync(kFull, incl, off);
    if (lane >= off) incl += v;
  }
  const int total = __shfl_sync(kFull, incl, 31);
  int base = 0;
  if (lane == 31 && total) base = atomicAdd(out_count, total);
  base = __shfl_sync(kFull, base, 31);
  if (!cnt) return;
  const int pixel = pixel_of_rank[k];
  const int16_t x = (int16_t)(pixel % width), y = (int16_t)(pixel / width);
  int o = base + incl - cnt;
  for (int j = 0; j < cnt; ++j, ++o) {
    DevEvent e;
    e.t = slab_t[(size_t)k * max_events + j];
    e.depth = -1.0f;
    e.rank = k;
    e.x = x;
    e.y = y;
    e.polarity = slab_p[(size_t)k * max_events + j];
    e.pad[0] = e.pad[1] = e.pad[2] = 0;
    out[o] = e;
  }
}

// Event-time depth re-trace (event_sensor.cu:51-59): a warp per event, its lanes on the pixel's sub-rays, so a packet
// is one pixel at one time; grid-stride over the device-side event count.  (32 events of different pixels and times in
// a packet, each lane its sub-rays one after the other, took 1.9 ms for 25 events at 16 sub-rays, and 0.32 ms for 225
// at one.)
struct DepthShared {
  int code[kStackSlots];
  float t[kStackSlots];
  float hit_t[32];
};
template <int kGeo>
__global__ void __launch_bounds__(128) event_depth_kernel(const __grid_constant__ SceneView S,
                                                          const dvs_optical_interval *ivs, int n_ivs,
                                                          DevEvent *events, const int32_t *count, int32_t *error,
                                                          unsigned long long *counters) {
  __shared__ DepthShared s_warp[kWarpsPerBlock];
  DepthShared &sh = s_warp[threadIdx.x >> 5];
  const int n = *count, lane = threadIdx.x & 31, ss2 = S.samples * S.samples;
  const int warps = gridDim.x * kWarpsPerBlock;
  unsigned primary = 0;
  for (int e = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); e < n; e += warps) {
    const double t = events[e].t;
    // first interval whose t1 >= t (the reference's forward scan, :54)
    int lo = 0, hi = n_ivs - 1;
    while (lo < hi) {
      int mid = (lo + hi) >> 1;
      if (t > ivs[mid].t1) lo = mid + 1; else hi = mid;
    }
    const CellPose pose = pose_at(ivs[lo], t);
    const int pixel = S.pixel_of_rank[events[e].rank];
    const int px_i = pixel % S.width, py_i = pixel / S.width;
    double depth = 0;
    int valid_depth = 0;
    bool bad = false;
    for (int r0 = 0; r0 < ss2; r0 += 32) {
      const bool live = r0 + lane < ss2;
      const int r = live ? r0 + lane : 0;
      const float3 ray[1] = {unit(rotate_ray(pose, f3(subray_x(S, px_i, r % S.samples),
                                                      -subray_y(S, py_i, r / S.samples), -1)))};
      const float3 origin[1] = {f3(pose.px, pose.py, pose.pz)};
      const bool lives[1] = {live};
      HitRecord hit[1];
      trace_nearest_packet_r<1, kGeo>(S, origin, ray, lives, sh.code, sh.t, hit);
      bad = bad || hit[0].hit < 0;
      sh.hit_t[lane] = live && hit[0].hit == 1 ? hit[0].t : -1.0f;
      __syncwarp();
      if (lane == 0)
        for (int i = 0; i < min(32, ss2 - r0); ++i)
          if (sh.hit_t[i] >= 0.0f) {  // in sub-ray order
            depth += sh.hit_t[i];
            ++valid_depth;
          }
      __syncwarp();
    }
    if (lane == 0) {
      if (bad) atomicOr(error, kErrOptical);
      events[e].depth = valid_depth ? float(depth / valid_depth) : -1.0f;
    }
    primary += ss2;
  }
  if (lane == 0 && counters && primary) atomicAdd(counters + kCntPrimary, (unsigned long long)primary);
}

__global__ void radiance_to_float_kernel(int n, const int32_t *pixel_of_rank, const double *radiance,
                                         const float *depth, float *image, float *depth_image) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int pixel = pixel_of_rank[k];
  image[pixel] = (float)radiance[k];
  if (depth_image) depth_image[pixel] = depth[k];
}

// Time-weighted exposure of a motion-blur frame (apps/main_cam_blur.cpp:66-73):
// per pixel, in pose order, acc += float(radiance of pose j) * weight[j].
__global__ void blur_accumulate_kernel(int n, int n_poses, const int32_t *pixel_of_rank, const double *radiance,
                                       const float *weights, float *image) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  float acc = 0.0f;
  for (int j = 0; j < n_poses; ++j) acc = acc + (float)radiance[(size_t)j * n + k] * __ldg(weights + j);
  image[pixel_of_rank[k]] = acc;
}

// Photon counts as the circuit kernels draw them, one per thread: generator 0
// is the reference's stream -- curand_init(seed, i, 0) and poisson_electrons,
// as the counts kernel of tests/test_sensor.cu:17-20 -- and generator 1 the
// precision mode's Philox stream of pixel i at the cell starting at cell_t0.
__global__ void poisson_draws_kernel(int generator, double lambda, unsigned seed, int n, double cell_t0,
                                     double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (generator == 0) {
    curandStateXORWOW_t rng;
    curand_init(seed, i, 0, &rng);
    out[i] = poisson_electrons(rng, lambda);
  } else {
    curandStatePhilox4_32_10_t ph = philox_at(seed, i, cell_t0);
    out[i] = poisson_electrons_philox(ph, (float)lambda);
  }
}

constexpr long long kResidentWarps = 2432;  // 152 SMs x 16 warps
inline int blocks(long long threads, int per_block) { return (int)((threads + per_block - 1) / per_block); }

}  // namespace

cudaError_t launch_poisson_draws(int generator, double lambda, unsigned seed, int n, double cell_t0, double *out,
                                 cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  poisson_draws_kernel<<<blocks(n, 128), 128, 0, s>>>(generator, lambda, seed, n, cell_t0, out);
  return cudaGetLastError();
}

// ---- launchers ----------------------------------------------------------------------
cudaError_t launch_hapke_const(const dvs_hapke &hapke, HapkeConst *out, cudaStream_t s) {
  hapke_const_kernel<<<1, 1, 0, s>>>(hapke, out);
  return cudaGetLastError();
}

cudaError_t launch_pose_from_state(const dvs_optical_state *state, CellPose *out, cudaStream_t s) {
  pose_from_state_kernel<<<1, 32, 0, s>>>(state, out);
  return cudaGetLastError();
}

cudaError_t launch_poses_from_states(const dvs_optical_state *states, int n, CellPose *out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  poses_from_states_kernel<<<blocks(n, 128), 128, 0, s>>>(states, n, out);
  return cudaGetLastError();
}

cudaError_t launch_blur_accumulate(int n, int n_poses, const int32_t *pixel_of_rank, const double *radiance,
                                   const float *weights, float *image, cudaStream_t s) {
  blur_accumulate_kernel<<<blocks(n, 128), 128, 0, s>>>(n, n_poses, pixel_of_rank, radiance, weights, image);
  return cudaGetLastError();
}

cudaError_t launch_cell_poses(const dvs_optical_interval *ivs, const Cell *cells, int n, CellPose *out,
                              cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  cell_poses_kernel<<<blocks(n, 128), 128, 0, s>>>(ivs, cells, n, out);
  return cudaGetLastError();
}

// Few poses: packets of sub-rays.  One sub-ray a pixel fills a packet with a block of 8 x 4 pixels; where so few pixels
// leave the GPU idle, narrower packets on more warps.
bool trace_by_pose(const SceneView &scene, int n_pix, int nc) {
  if (nc >= 8) return false;
  return scene.samples > 1 || (long long)n_pix * nc < 32 * kResidentWarps;
}
PoseShape pose_item_shape(int n_pix, int nc, int ss2, bool scattered) {
  PoseShape s{1, 0, 0};
  while ((1 << s.lanes_log2) < ss2 && s.lanes_log2 < 5) ++s.lanes_log2;
  const int per_packet = 32 >> s.lanes_log2, runs = (ss2 + 31) / 32;
  // pixels of an item: a packet's, then more for the beam while every SM has items (scattered pixels share no beam)
  const int most = std::min(32, kPoseTerms / ((1 << s.lanes_log2) + 1));
  const auto items = [&](int pixels) { return (long long)((n_pix + pixels - 1) / pixels) * nc; };
  const int limit = scattered ? per_packet : most;
  while (2 * s.pixels <= limit && items(2 * s.pixels) >= 2 * kResidentWarps && s.pixels * runs < 64 * per_packet)
    s.pixels *= 2;
  // one walk for the item pays from 8 packets on, or where the item is itself one narrow packet (the walk takes four
  // nodes at a time and sorts once: 160x120 frames with 4 sub-rays 0.29 -> 0.20 ms); 4 packets over 32 pixels lose 8 %
  s.beam = scattered ? s.pixels == 1 : s.pixels <= 4 || (s.pixels + per_packet - 1) / per_packet * runs >= 8;
  return s;
}

namespace {
template <int kGeo>
void trace_list_geo(const SceneView &scene, int n_pix, const int32_t *rank_list, const CellPose *poses, int c0, int nc,
                    int cw_log2, double *radiance, float *depth, unsigned long long *counters, cudaStream_t s) {
  if (trace_by_pose(scene, n_pix, nc)) {
    const PoseShape shape = pose_item_shape(n_pix, nc, scene.samples * scene.samples, rank_list != nullptr);
    const int grid = blocks((long long)((n_pix + shape.pixels - 1) / shape.pixels) * nc * 32, 128);
    if (depth)
      trace_poses_kernel<kRadianceDepth, kGeo><<<grid, 128, 0, s>>>(scene, n_pix, rank_list, poses, c0, nc, shape,
                                                                    radiance, depth, counters);
    else
      trace_poses_kernel<kRadiance, kGeo><<<grid, 128, 0, s>>>(scene, n_pix, rank_list, poses, c0, nc, shape, radiance,
                                                               nullptr, counters);
    return;
  }
  const int ss2 = scene.samples * scene.samples;
  const int rays = trace_rays(scene, n_pix, nc, cw_log2, rank_list != nullptr);
  const ItemShape shape = trace_item_shape(n_pix, nc, cw_log2, ss2, rays, rank_list != nullptr);
  const int grid = blocks(trace_job_items(n_pix, nc, shape) * 32, 128);
#define DVS_TRACE_LAUNCH(MODE, RAYS, BEAM)                                                                        \
  trace_cells_kernel<MODE, RAYS, kGeo, BEAM><<<grid, 128, 0, s>>>(scene, n_pix, rank_list, poses, c0, nc, shape, \
                                                                  radiance, depth, counters)
#define DVS_TRACE_MODE(MODE)                            \
  do {                                                  \
    if constexpr (kGeo == kGeoReference)                \
      if (rays == 4) { DVS_TRACE_LAUNCH(MODE, 4, false); return; } \
    if (rays == 2) DVS_TRACE_LAUNCH(MODE, 2, false);    \
    else if (shape.beam) DVS_TRACE_LAUNCH(MODE, 1, true); \
    else DVS_TRACE_LAUNCH(MODE, 1, false);              \
  } while (0)
  if (depth) DVS_TRACE_MODE(kRadianceDepth);
  else DVS_TRACE_MODE(kRadiance);
#undef DVS_TRACE_MODE
#undef DVS_TRACE_LAUNCH
}
}  // namespace

cudaError_t launch_trace_list(const SceneView &scene, int n_pix, const int32_t *rank_list, const CellPose *poses,
                              int c0, int nc, int cw_log2, double *radiance, float *depth, unsigned long long *counters,
                              cudaStream_t s) {
  if (n_pix <= 0 || nc <= 0) return cudaSuccess;
  switch (scene.geometry) {
    case kGeoHalfBounds:
      trace_list_geo<kGeoHalfBounds>(scene, n_pix, rank_list, poses, c0, nc, cw_log2, radiance, depth, counters, s);
      break;
    case kGeoWatertight:
      trace_list_geo<kGeoWatertight>(scene, n_pix, rank_list, poses, c0, nc, cw_log2, radiance, depth, counters, s);
      break;
    case kGeoHalfBounds | kGeoWatertight:
      trace_list_geo<kGeoHalfBounds | kGeoWatertight>(scene, n_pix, rank_list, poses, c0, nc, cw_log2, radiance,
                                                      depth, counters, s);
      break;
    default:
      trace_list_geo<kGeoReference>(scene, n_pix, rank_list, poses, c0, nc, cw_log2, radiance, depth, counters, s);
  }
  return cudaGetLastError();
}

cudaError_t launch_trace_cells(const SceneView &scene, int n_pix, const CellPose *poses, int c0, int nc, int cw_log2,
                               double *radiance, float *depth, unsigned long long *counters, cudaStream_t s) {
  return launch_trace_list(scene, n_pix, nullptr, poses, c0, nc, cw_log2, radiance, depth, counters, s);
}

cudaError_t launch_init_pixels(int n, const int32_t *pixel_of_rank, const double *radiance, PixelParams p,
                               PhotoParams photo, double stddev, double minimum, unsigned seed, CircuitState st,
                               int32_t *error, cudaStream_t s) {
  if (photo.philox)
    init_pixels_kernel<curandStatePhilox4_32_10_t><<<blocks(n, 128), 128, 0, s>>>(n, pixel_of_rank, radiance, p, photo,
                                                                                stddev, minimum, seed, st, error);
  else
    init_pixels_kernel<curandStateXORWOW_t><<<blocks(n, 128), 128, 0, s>>>(n, pixel_of_rank, radiance, p, photo, stddev,
                                                                         minimum, seed, st, error);
  return cudaGetLastError();
}

cudaError_t launch_circuit_list(int n, const int32_t *rank_list, const Cell *cells, int c0, int nc,
                                const double *radiance, PixelParams p, PhotoParams photo, int max_events,
                                CircuitState st, int32_t *ev_count, double *slab_t, int8_t *slab_p, int32_t *error,
                                unsigned long long *counters, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (photo.fp32_circuit && photo.philox)
    circuit_kernel<true, true><<<blocks(n, 128), 128, 0, s>>>(n, rank_list, cells, c0, nc, radiance, p, photo,
                                                              max_events, st, ev_count, slab_t, slab_p, error, counters);
  else if (photo.fp32_circuit)
    circuit_kernel<true, false><<<blocks(n, 128), 128, 0, s>>>(n, rank_list, cells, c0, nc, radiance, p, photo,
                                                               max_events, st, ev_count, slab_t, slab_p, error, counters);
  else
    circuit_kernel<false, false><<<blocks(n, 128), 128, 0, s>>>(n, rank_list, cells, c0, nc, radiance, p, photo,
                                                                max_events, st, ev_count, slab_t, slab_p, error,
                                                                counters);
  return cudaGetLastError();
}

// A Philox draw depends on its pixel and cell alone.  With few pixels the
// circuit's threads, one a pixel, cannot hide a cell's chain of draw and receptor
// step, so the draws of all cells go ahead on a thread each: 64 cells of 64x48
// pixels 93 -> 68 us, of 128x96 95 -> 76.  The gain shrinks to 4 us at 256x192 and
// is a loss of 8 at 320x240 (110 -> 118), so the line lies below both, at 38,912
// pixels: two warps a scheduler.  (Reset noise continues a cell's stream after its
// draw and keeps the draw in the circuit.)
bool circuit_draws_ahead(int n, const PixelParams &p, const PhotoParams &photo) {
  return photo.philox && photo.chunk_f32 && photo.shot_noise && p.reset_noise_std == 0 && n < kResidentWarps * 16;
}

cudaError_t launch_circuit(int n, const Cell *cells, int c0, int nc, double *radiance, PixelParams p,
                           PhotoParams photo, int max_events, CircuitState st, int32_t *ev_count, double *slab_t,
                           int8_t *slab_p, int32_t *error, unsigned long long *counters, cudaStream_t s) {
  if (circuit_draws_ahead(n, p, photo)) {
    philox_draws_kernel<<<blocks((long long)n * nc, 128), 128, 0, s>>>(n, cells, c0, nc, st.pixel, photo,
                                                                       reinterpret_cast<float *>(radiance));
    photo.drawn = 1;
  }
  return launch_circuit_list(n, nullptr, cells, c0, nc, radiance, p, photo, max_events, st, ev_count, slab_t, slab_p,
                             error, counters, s);
}

cudaError_t launch_emit_events(int n, const int32_t *pixel_of_rank, int width, int max_events, const int32_t *ev_count,
                               const double *slab_t, const int8_t *slab_p, DevEvent *out, int32_t *out_count,
                               cudaStream_t s) {
  emit_events_kernel<<<blocks(n, 128), 128, 0, s>>>(n, pixel_of_rank, width, max_events, ev_count, slab_t, slab_p,
                                                    out, out_count);
  return cudaGetLastError();
}

cudaError_t launch_event_depth(const SceneView &scene, const dvs_optical_interval *ivs, int n_ivs, DevEvent *events,
                               const int32_t *count, int32_t *error, unsigned long long *counters, cudaStream_t s) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  switch (scene.geometry) {
    case kGeoHalfBounds:
      event_depth_kernel<kGeoHalfBounds><<<sms * 4, 128, 0, s>>>(scene, ivs, n_ivs, events, count, error, counters);
      break;
    case kGeoWatertight:
      event_depth_kernel<kGeoWatertight><<<sms * 4, 128, 0, s>>>(scene, ivs, n_ivs, events, count, error, counters);
      break;
    case kGeoHalfBounds | kGeoWatertight:
      event_depth_kernel<kGeoHalfBounds | kGeoWatertight><<<sms * 4, 128, 0, s>>>(scene, ivs, n_ivs, events, count,
                                                                                 error, counters);
      break;
    default:
      event_depth_kernel<kGeoReference><<<sms * 4, 128, 0, s>>>(scene, ivs, n_ivs, events, count, error, counters);
  }
  return cudaGetLastError();
}

namespace {
template <int kMode, int kRays, int kGeo>
cudaError_t preload_cells() {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, trace_cells_kernel<kMode, kRays, kGeo, false>);
  if constexpr (kRays == 1)
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, trace_cells_kernel<kMode, kRays, kGeo, true>);
  return e;
}
template <int kGeo>
cudaError_t preload_camera_geo() {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, trace_poses_kernel<kRadianceDepth, kGeo>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, trace_poses_kernel<kRadiance, kGeo>);
  if (e == cudaSuccess) e = preload_cells<kRadianceDepth, 1, kGeo>();
  if (e == cudaSuccess) e = preload_cells<kRadianceDepth, 2, kGeo>();
  if (e == cudaSuccess) e = preload_cells<kRadiance, 1, kGeo>();
  if (e == cudaSuccess) e = preload_cells<kRadiance, 2, kGeo>();
  if constexpr (kGeo == kGeoReference) {
    if (e == cudaSuccess) e = preload_cells<kRadianceDepth, 4, kGeo>();
    if (e == cudaSuccess) e = preload_cells<kRadiance, 4, kGeo>();
  }
  return e;
}
}  // namespace

cudaError_t preload_camera_kernels(int geometry) {
  // cudaFuncGetAttributes loads a kernel that lazy module loading has not
  // loaded yet, so a later launch of it allocates nothing
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, radiance_to_float_kernel);
  if (e != cudaSuccess) return e;
  switch (geometry) {
    case kGeoHalfBounds: return preload_camera_geo<kGeoHalfBounds>();
    case kGeoWatertight: return preload_camera_geo<kGeoWatertight>();
    case kGeoHalfBounds | kGeoWatertight: return preload_camera_geo<kGeoHalfBounds | kGeoWatertight>();
    default: return preload_camera_geo<kGeoReference>();
  }
}

cudaError_t launch_radiance_to_float(int n, const int32_t *pixel_of_rank, const double *radiance, const float *depth,
                                     float *image, float *depth_image, cudaStream_t s) {
  radiance_to_float_kernel<<<blocks(n, 128), 128, 0, s>>>(n, pixel_of_rank, radiance, depth, image, depth_image);
  return cudaGetLastError();
}

}  // namespace dvsgb
