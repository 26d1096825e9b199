// Adaptive optical refinement on the GB300 path (replaces the reference's
// OpticalSampler::refine / prepare_exact_cells and EventSensor::
// process_adaptive kernels: src/cuda/optical_sampler.cu:25-138,
// src/cuda/event_sensor.cu:88-150).
//
// Per pixel, the radiance over a batch window is probed at 0, 1/4, 1/2, 3/4
// and 1 and bisected until a segment's linear interpolation predicts the
// receptor voltage within 1e-3 of the pixel's smaller threshold; segments
// that stay unresolved at the circuit-cell scale are marked for exact
// tracing of the cells inside them.  The circuit then integrates every
// native cell from the interpolated (or exactly traced) radiance.
//
// GB300 mapping: a warp per pixel, as the reference, but with the pixel's
// pending segments one per lane (refine_kernel).  The probe value is the
// pixel's serial sub-ray mean, the same double the reference's warp_radiance
// returns.
#include <cstdint>
#include <cuda_runtime.h>

#include "kernels.h"
#include "device_optics.cuh"
#include "device_circuit.cuh"

namespace dvsgb {
namespace {

constexpr int kRefineStack = 16;  // optical_sampler.cu:43

// native_pose (optical_sampler.cu:26-30): the interval holding t.
__device__ __forceinline__ CellPose native_pose(const dvs_optical_interval *ivs, int count, double t) {
  int lo = 0, hi = count - 1;
  while (lo < hi) {
    const int m = (lo + hi) / 2;
    if (t > ivs[m].t1) lo = m + 1; else hi = m;
  }
  return pose_at(ivs[lo], t);
}

__device__ __forceinline__ double segment_fraction(const OpticalKnot *values, int a) { return fabs(values[a].fraction); }

// The poses of the five initial probes (0, 1/4, 1/2, 3/4, 1 of the window).
__global__ void probe_poses_kernel(const dvs_optical_interval *ivs, int n_ivs, double start, double end,
                                   CellPose *out) {
  const int j = threadIdx.x;
  if (j < 5) out[j] = native_pose(ivs, n_ivs, start + (end - start) * j * .25);
}

// refine_pixels (optical_sampler.cu:39-84), one warp per pixel.  The five
// initial probes come traced by the native trace kernel (initial[j * n +
// rank]: every pixel is probed at the same five times, so they are five
// circuit cells of a temporal warp packet); the bisection probes, which only
// some pixels need, are traced here.
//
// The lanes hold the pixel's pending segments in time order: the reference's
// depth-first stack, opened ahead.  A segment's verdict depends on the segment
// and on how many wait behind it in that stack (`behind`, which a split hands
// on: +1 to the left half), not on when it is reached, so every iteration
// judges all pending segments at once (the FP64 receptor steps, one segment
// per lane), emits the finished ones at the front in order, and splits up to
// kAhead pending segments: two probes each, their poses one per lane, their
// sub-rays 32 to a packet through the pixel's beam.  Knots, fallbacks and
// counters are the depth-first walk's: an overflow of the knot capacity takes
// back the splits that walk would not have reached, their rays and their
// errors.  Those are the splits of segments that lie behind the overflow, so
// each split's tally goes with the leftmost of its pending descendants.
//
// Bound by the latency of the probes' packets and the FP64 pipe of the
// verdicts.  One pixel per lane instead (32 pixels in lock-step, each lane
// its sub-rays one after the other) took 312 ms for 120 x 90 pixels and
// 200 horizons of 10 us at 16 sub-rays, every probe a packet of 32 times.
constexpr int kAhead = 16;        // pending segments beyond which only the first is split: with its at most
                                  // kRefineStack - 1 further left halves the list stays within 32 lanes
constexpr int kProbeRays = 16;    // sub-rays of a probe traced and summed at a time
struct RefineShared {
  int code[kStackSlots];
  float t[kStackSlots];
  Beam beam;
  CellPose pose[32];
  double term[32][kProbeRays + 1];  // [probe][sub-ray], rows apart in the banks
  double seg[5][32];
  unsigned long long tally[32];
  int behind[32], verdict[32];
  unsigned char traced[32][kProbeRays + 4];  // rays of term's sub-ray (1, or 2 with its shadow ray), kProbeBad
};
constexpr int kProbeBad = 4;
// a tally counts rays, and above them probes that overflowed or are not finite
constexpr int kTallyBadShift = 40;
enum : int { kUndecided = 0, kSmooth = 1, kExact = 2, kSplit = 3 };

template <int kGeo>
__global__ void __launch_bounds__(128, 4)
    refine_kernel(const __grid_constant__ SceneView S, int n, const dvs_optical_interval *ivs, int n_ivs, double start,
                  double end, PhotoParams photo, double tolerance, CircuitState st, double charge, int capacity,
                  const double *initial_radiance, OpticalKnot *knots, int32_t *counts, unsigned long long *ref_stats,
                  int32_t *error, unsigned long long *counters) {
  extern __shared__ __align__(16) unsigned char refine_shared[];
  RefineShared &sh = reinterpret_cast<RefineShared *>(refine_shared)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int rank = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (rank >= n) return;  // warp-uniform
  const int pixel = S.pixel_of_rank[rank];
  const int px_i = pixel % S.width, py_i = pixel / S.width, ss2 = S.samples * S.samples;
  bool bad = false;
  unsigned long long traced = 0, tally = 0;  // of this lane's probes; of the splits that go with segment `lane`
  double initial[5];
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    initial[j] = initial_radiance[(size_t)j * n + rank];
    if (!isfinite(initial[j])) bad = true;
  }
  OpticalKnot *out = knots + (size_t)rank * capacity;
  const double x0 = exp(st.receptor_log[rank]), inv_charge = 1.0 / charge;
  const double budget = 1e-3 * fmin(st.threshold_pos[rank], st.threshold_neg[rank]);  // kOpticalVoltageThresholdFraction
  if (lane == 0) out[0] = {0, initial[0]};
  // lane i: pending segment i
  double a = 0, b = .5, left = initial[0], middle = initial[1], right = initial[2];
  int behind = 1, verdict = kUndecided;
  if (lane == 1) {
    a = .5;
    b = 1;
    left = initial[2];
    middle = initial[3];
    right = initial[4];
    behind = 0;
  }
  int pending = 2, written = 1, splits = 0, exact_segments = 0, not_reached = 0;
  bool fallback = false, no_beam = true;
  BeamLists lists{kNoList, kNoList, 0};
  while (pending > 0) {
    if (lane < pending && verdict == kUndecided) {
      const double actual = middle * photo.electrons_per_radiance + photo.dark_electrons;
      const double estimate = (left + right) * .5 * photo.electrons_per_radiance + photo.dark_electrons;
      const double leaf_duration = (b - a) * (end - start);
      // |u(actual) - u(estimate)| from the receptors themselves: one log for both
      const double voltage_error = fabs(log(receptor_step(x0, fmax(0.0, actual), leaf_duration * inv_charge) /
                                            receptor_step(x0, fmax(0.0, estimate), leaf_duration * inv_charge)));
      bool smooth = voltage_error <= budget;
      if (smooth && !(fmax(actual, estimate) * leaf_duration < 1.0))
        smooth = fabs(log(fmax(1e-30, actual) / fmax(1e-30, estimate))) <= tolerance;
      if (smooth)
        verdict = kSmooth;
      else if ((b - a) * (end - start) <= photo.integration_step || behind + 2 > kRefineStack)
        verdict = kExact;  // unresolved at the electrical sampling scale: exact tracing
      else
        verdict = kSplit;
    }
    __syncwarp();
    const unsigned to_split = __ballot_sync(kFull, lane < pending && verdict == kSplit);
    const int done = to_split ? __ffs(to_split) - 1 : pending;  // finished segments at the front
    if (done > 0) {
      const unsigned two = __ballot_sync(kFull, lane < done && verdict == kSmooth);
      const unsigned one = __ballot_sync(kFull, lane < done && verdict == kExact);
      const int at = written + 2 * __popc(two & below) + __popc(one & below);
      const bool over = lane < done && (verdict == kSmooth ? at + 2 > capacity : at >= capacity);
      const unsigned overs = __ballot_sync(kFull, over);
      const int emit = overs ? __ffs(overs) - 1 : done;
      const unsigned emitted = emit >= 32 ? kFull : (1u << emit) - 1u;
      if (lane < emit) {
        if (verdict == kSmooth) {
          out[at] = {(a + b) * .5, middle};
          out[at + 1] = {b, right};
        } else {
          out[at] = {-b, right};
        }
      }
      written += 2 * __popc(two & emitted) + __popc(one & emitted);
      exact_segments += __popc(one & emitted);
      if (overs) {
        fallback = true;
        not_reached = pending - 1 - emit - __shfl_sync(kFull, behind, emit);
        if (lane > emit && lane < pending) traced -= tally;  // modulo 2^64; the warp's sum is not negative
        break;
      }
      pending -= done;
      const int from = (lane + done) & 31;
      a = __shfl_sync(kFull, a, from);
      b = __shfl_sync(kFull, b, from);
      left = __shfl_sync(kFull, left, from);
      middle = __shfl_sync(kFull, middle, from);
      right = __shfl_sync(kFull, right, from);
      behind = __shfl_sync(kFull, behind, from);
      verdict = __shfl_sync(kFull, verdict, from);
      tally = __shfl_sync(kFull, tally, from);
    }
    if (pending == 0) break;
    // the first pending segment splits; others while the list stays within kAhead
    const unsigned wants = to_split >> done;
    const int count = max(1, min(__popc(wants), kAhead - pending));
    const bool mine = ((wants >> lane) & 1u) && __popc(wants & below) < count;
    const unsigned chosen = __ballot_sync(kFull, mine);
    const int slot = __popc(chosen & below);
    if (no_beam) {  // the first split: the pixel's beam over the window, from the corners at the initial probe times
      no_beam = false;
      const int last = S.samples - 1, j = min(lane >> 2, 4);
      const CellPose pose = native_pose(ivs, n_ivs, start + (end - start) * j * .25);
      const float3 o = f3(pose.px, pose.py, pose.pz), l = inverse_direction(f3(pose.lx, pose.ly, pose.lz));
      const float3 d = unit(rotate_ray(pose, f3(subray_x(S, px_i, lane & 1 ? last : 0),
                                                -subray_y(S, py_i, lane & 2 ? last : 0), -1)));
      lists = close_beam<kGeo>(S, o, o, d, d, l, l, 0.05f, sh.beam, sh.code);
    }
    if (mine) {
      sh.seg[0][slot] = a;
      sh.seg[1][slot] = b;
    }
    __syncwarp();
    const int probes = 2 * count;
    if (lane < probes) {
      const double pa = sh.seg[0][lane >> 1], pb = sh.seg[1][lane >> 1], mid = (pa + pb) * .5;
      const double t = lane & 1 ? start + (end - start) * (mid + pb) * .5 : start + (end - start) * (pa + mid) * .5;
      sh.pose[lane] = native_pose(ivs, n_ivs, t);
    }
    __syncwarp();
    double sum = 0;
    unsigned long long probe = 0;
    bool probe_bad = false;
    for (int r0 = 0; r0 < ss2; r0 += kProbeRays) {
      const int m = min(kProbeRays, ss2 - r0), total = probes * m;
      for (int q0 = 0; q0 < total; q0 += 32) {
        const int q = min(q0 + lane, total - 1), k = q / m, r = r0 + q - k * m;
        const bool live = q0 + lane < total;
        const CellPose pose = sh.pose[k];
        const RaySample s = sample_ray<kGeo, true>(S, subray_x(S, px_i, r % S.samples),
                                                   subray_y(S, py_i, r / S.samples), pose, live, sh.code,
                                                   sh.t, sh.beam, lists);
        if (live) {
          sh.term[k][q - k * m] = s.term;
          sh.traced[k][q - k * m] = (unsigned char)((s.lit ? 2 : 1) | (s.overflow ? kProbeBad : 0));
        }
      }
      __syncwarp();
      if (lane < probes)
        for (int i = 0; i < m; ++i) {
          sum += sh.term[lane][i];  // in sub-ray order, as the pixel sample's sum
          const unsigned t = sh.traced[lane][i];
          probe += t & 3u;
          probe_bad |= (t & kProbeBad) != 0;
        }
      __syncwarp();
    }
    sum /= ss2;
    if (lane < probes && (probe_bad || !isfinite(sum))) probe += 1ull << kTallyBadShift;
    traced += probe;
    // the list with each chosen segment replaced by its halves
    const double left_mid = __shfl_sync(kFull, sum, (2 * slot) & 31), right_mid = __shfl_sync(kFull, sum, (2 * slot + 1) & 31);
    const unsigned long long spent = __shfl_sync(kFull, probe, (2 * slot) & 31) + __shfl_sync(kFull, probe, (2 * slot + 1) & 31);
    const int to = lane + slot;
    if (lane < pending) {
      const double mid = (a + b) * .5;
      sh.seg[0][to] = a;
      sh.seg[1][to] = mine ? mid : b;
      sh.seg[2][to] = left;
      sh.seg[3][to] = mine ? left_mid : middle;
      sh.seg[4][to] = mine ? middle : right;
      sh.behind[to] = mine ? behind + 1 : behind;
      sh.verdict[to] = mine ? kUndecided : verdict;
      sh.tally[to] = mine ? tally + spent : tally;
      if (mine) {
        sh.seg[0][to + 1] = mid;
        sh.seg[1][to + 1] = b;
        sh.seg[2][to + 1] = middle;
        sh.seg[3][to + 1] = right_mid;
        sh.seg[4][to + 1] = right;
        sh.behind[to + 1] = behind;
        sh.verdict[to + 1] = kUndecided;
        sh.tally[to + 1] = 0;
      }
    }
    __syncwarp();
    pending += count;
    splits += count;
    a = sh.seg[0][lane];
    b = sh.seg[1][lane];
    left = sh.seg[2][lane];
    middle = sh.seg[3][lane];
    right = sh.seg[4][lane];
    behind = sh.behind[lane];
    verdict = sh.verdict[lane];
    tally = sh.tally[lane];
    __syncwarp();
  }
#pragma unroll
  for (int k = 16; k; k >>= 1) traced += __shfl_xor_sync(kFull, traced, k);
  if (bad || traced >> kTallyBadShift) atomicOr(error, kErrOptical);
  if (lane == 0) {
    counts[rank] = fallback ? -1 : written;
    atomicAdd(ref_stats + kRefTraced, 5ull + 2ull * (unsigned)(splits - not_reached));
    if (fallback) atomicAdd(ref_stats + kRefFallback, 1ull);
    else atomicMax(ref_stats + kRefMaxKnots, (unsigned long long)written);
    if (exact_segments) atomicAdd(ref_stats + kRefExactSegments, (unsigned long long)exact_segments);
  }
  if (lane == 0 && counters) atomicAdd(counters + kCntPrimary, traced & ((1ull << kTallyBadShift) - 1));
}

// identify_exact_cells (optical_sampler.cu:114-131): cells whose midpoint falls
// in a marked segment are queued for exact tracing.
__global__ void identify_exact_kernel(int n, const Cell *cells, int n_cells, double start, double end,
                                      const OpticalKnot *knots, int32_t *knot_counts, int capacity,
                                      int32_t *exact_cells, int32_t *exact_counts, int32_t *queue, int32_t *total,
                                      unsigned long long *ref_stats) {
  const int rank = blockIdx.x * blockDim.x + threadIdx.x;
  if (rank >= n) return;
  exact_counts[rank] = 0;
  const int size = knot_counts[rank];
  if (size < 0) return;
  const OpticalKnot *values = knots + (size_t)rank * capacity;
  int a = 0, used = 0;
  for (int c = 0; c < n_cells; ++c) {
    const double fraction = ((cells[c].t0 + cells[c].t1) * .5 - start) / (end - start);
    while (a + 2 < size && fraction > fabs(values[a + 1].fraction)) ++a;
    if (values[a + 1].fraction < 0) {
      if (used == capacity) {
        knot_counts[rank] = -1;
        atomicAdd(ref_stats + kRefFallback, 1ull);
        return;
      }
      exact_cells[(size_t)rank * capacity + used++] = c;
    }
  }
  exact_counts[rank] = used;
  if (!used) return;
  const int offset = atomicAdd(total, used);
  for (int j = 0; j < used; ++j) queue[offset + j] = rank * capacity + j;
}

// sample_exact_queries (optical_sampler.cu:132-138): one queued cell per lane,
// grid-stride over the device-side queue length.
template <int kGeo>
__global__ void __launch_bounds__(128) sample_exact_kernel(const __grid_constant__ SceneView S, const CellPose *poses,
                                                           const int32_t *exact_cells, const int32_t *queue,
                                                           const int32_t *total, int capacity, double *exact_radiance,
                                                           int32_t *error, unsigned long long *counters) {
  __shared__ int s_code[4][kStackSlots];
  __shared__ float s_t[4][kStackSlots];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int count = *total;
  const int stride = gridDim.x * blockDim.x;
  for (int base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; base < count; base += stride) {
    const int q = base + lane;
    const bool active = q < count;
    const int slot = active ? queue[q] : 0;
    const int rank = slot / capacity;
    const int pixel = active ? S.pixel_of_rank[rank] : 0;
    const CellPose pose = poses[active ? exact_cells[slot] : 0];
    const PixelSample s = sample_pixel_group<kRadiance, 1, kGeo, false>(S, pixel, active, pose, s_code[wib], s_t[wib],
                                                                        nullptr, nullptr, nullptr);
    if (active) {
      if (!s.valid || !isfinite(s.radiance)) atomicOr(error, kErrOptical);
      exact_radiance[slot] = s.radiance;
    }
    const unsigned r = __reduce_add_sync(kFull, s.primary + s.shadow);
    if (lane == 0 && counters) atomicAdd(counters + kCntPrimary, (unsigned long long)r);
  }
}

// integrate_optical_knots (event_sensor.cu:88-114): every native cell from the
// knots (or its exactly traced radiance); events carry no depth.  Bound by the
// FP64 pipe: the cells' window fractions, the same for every pixel, are
// formed 32 at a time, shared out over the lanes (in every thread, with its quotient by the
// window, they made 120 x 90 pixels x 200 horizons of 10 us 67.1 ms instead of 62.5).
__global__ void __launch_bounds__(128) integrate_knots_kernel(int n, const Cell *cells, int n_cells, double start,
                                                              double end, const OpticalKnot *knots,
                                                              const int32_t *knot_counts, int capacity,
                                                              const int32_t *exact_cells, const double *exact_radiance,
                                                              const int32_t *exact_counts, PixelParams p,
                                                              PhotoParams photo, int max_events, CircuitState st,
                                                              int32_t *ev_count, double *slab_t, int8_t *slab_p,
                                                              int32_t *error) {
  __shared__ double s_fraction[4][32];
  double *fractions = s_fraction[threadIdx.x >> 5];
  const int rank = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const bool mine = rank < n && knot_counts[rank] >= 0;
  const unsigned team = __ballot_sync(kFull, mine);  // the lanes with a pixel
  if (!mine) return;
  const int member = __popc(team & ((1u << lane) - 1u)), members = __popc(team);
  const OpticalKnot *values = knots + (size_t)rank * capacity;
  const int size = knot_counts[rank];
  const int n_exact = exact_counts ? exact_counts[rank] : 0;
  const int32_t *my_exact = exact_cells + (size_t)rank * capacity;
  const double *my_exact_rad = exact_radiance + (size_t)rank * capacity;
  CircuitRun run = circuit_begin(st, rank, p);
  curandStateXORWOW_t rng = st.rng[rank];
  double *my_t = slab_t + (size_t)rank * max_events;
  int8_t *my_p = slab_p + (size_t)rank * max_events;
  int a = 0, exact_index = 0, count = 0, failed = 0;
  // the segment [a, a + 1] of the knots: its left end and light, its length and the light's change over it
  double left = segment_fraction(values, 0), right = segment_fraction(values, 1);
  double from = values[0].radiance, change = values[1].radiance - from;
  double length = right - left, inv_length = 1.0 / length;
  for (int c0 = 0; c0 < n_cells; c0 += 32) {
    const int tile = min(32, n_cells - c0);
    for (int i = member; i < tile; i += members)
      fractions[i] = ((cells[c0 + i].t0 + cells[c0 + i].t1) * .5 - start) / (end - start);
    __syncwarp(team);
    for (int c = c0; !failed && c < c0 + tile; ++c) {
      const Cell cell = cells[c];
      const double fraction = fractions[c - c0];
      if (a + 2 < size && fraction > right) {
        do {
          ++a;
          right = segment_fraction(values, a + 1);
        } while (a + 2 < size && fraction > right);
        left = segment_fraction(values, a);
        from = values[a].radiance;
        change = values[a + 1].radiance - from;
        length = right - left;
        inv_length = 1.0 / length;
      }
      double light = from + change * quotient(fraction - left, length, inv_length);
      if (exact_index < n_exact && my_exact[exact_index] == c) light = my_exact_rad[exact_index++];
      double rate = (positive(light) ? light : 0.0) * photo.electrons_per_radiance + photo.dark_electrons;
      if (photo.shot_noise) rate = quotient(poisson_electrons(rng, rate * cell.len), cell.len, cell.inv_len);
      const int emitted = circuit_cell(run, p, rate, cell, my_t + count, my_p + count, max_events - count, rng);
      if (emitted == -1) failed = kErrCapacity;
      else if (emitted == -2) failed = kErrStalled;
      else count += emitted;
    }
    __syncwarp(team);
  }
  circuit_end(run, st, rank);
  st.rng[rank] = rng;
  if (failed) {
    atomicOr(error, failed);
    ev_count[rank] = -1;
  } else {
    ev_count[rank] = count;
  }
}

// compact_fallback (event_sensor.cu:116-118).
__global__ void compact_fallback_kernel(int n, const int32_t *knot_counts, int32_t *list, int32_t *total) {
  const int rank = blockIdx.x * blockDim.x + threadIdx.x;
  if (rank < n && knot_counts[rank] < 0) list[atomicAdd(total, 1)] = rank;
}

// advance_mean_probes (event_sensor.cu:138-150): receptor driven by exact and
// by knot-interpolated light for the probe pixels, over one cell chunk.
__global__ void advance_probes_kernel(int n_probes, const int32_t *probe_ranks, const Cell *cells, int c0, int nc,
                                      const double *light, const OpticalKnot *knots, const int32_t *knot_counts,
                                      int capacity, double start, double end, PhotoParams photo, double charge,
                                      double *probe_state) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_probes) return;
  const int rank = probe_ranks[i];
  const OpticalKnot *values = knots + (size_t)rank * capacity;
  double ex = probe_state[2 * i], ca = probe_state[2 * i + 1];
  for (int c = 0; c < nc; ++c) {
    const Cell cell = cells[c0 + c];
    const double exact = light[(size_t)c * n_probes + i];
    double cached = exact;
    if (knot_counts[rank] >= 0) {
      int a = 0;
      const double fraction = ((cell.t0 + cell.t1) * .5 - start) / (end - start);
      while (a + 2 < knot_counts[rank] && fraction > fabs(values[a + 1].fraction)) ++a;
      const double weight =
          (fraction - fabs(values[a].fraction)) / (fabs(values[a + 1].fraction) - fabs(values[a].fraction));
      if (values[a + 1].fraction >= 0) cached = values[a].radiance + (values[a + 1].radiance - values[a].radiance) * weight;
    }
    ex = receptor_log_at(ex, exact * photo.electrons_per_radiance + photo.dark_electrons, cell.t1 - cell.t0, charge);
    ca = receptor_log_at(ca, fmax(0.0, cached) * photo.electrons_per_radiance + photo.dark_electrons,
                         cell.t1 - cell.t0, charge);
  }
  probe_state[2 * i] = ex;
  probe_state[2 * i + 1] = ca;
}

__global__ void capture_probes_kernel(int n_probes, const int32_t *probe_ranks, const double *receptor_log,
                                      double *probe_state) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_probes) return;
  const double u = receptor_log[probe_ranks[i]];
  probe_state[2 * i] = u;
  probe_state[2 * i + 1] = u;
}

inline int blocks_of(long long threads, int per_block) { return (int)((threads + per_block - 1) / per_block); }
int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 1;
}

}  // namespace

cudaError_t launch_refine(const SceneView &scene, int n, const dvs_optical_interval *ivs, int n_ivs, double start,
                          double end, PhotoParams photo, double tolerance, CircuitState st, double charge,
                          int capacity, CellPose *probe_poses, double *probe_radiance, OpticalKnot *knots,
                          int32_t *counts, unsigned long long *ref_stats, int32_t *error,
                          unsigned long long *counters, cudaStream_t s) {
  // the five initial probes of every pixel: five cells of the native trace
  // kernel (8 cells per warp packet: 4 pixels x 5 probe times)
  probe_poses_kernel<<<1, 32, 0, s>>>(ivs, n_ivs, start, end, probe_poses);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = launch_trace_cells(scene, n, probe_poses, 0, 5, 3, probe_radiance, nullptr, counters, s);
  if (e != cudaSuccess) return e;
#define DVS_REFINE(G)                                                                                              \
  do {                                                                                                             \
    e = cudaFuncSetAttribute(refine_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);          \
    if (e != cudaSuccess) return e;                                                                                \
    refine_kernel<G><<<blocks_of(n, 4), 128, shared, s>>>(scene, n, ivs, n_ivs, start, end, photo, tolerance, st,  \
                                                          charge, capacity, probe_radiance, knots, counts,         \
                                                          ref_stats, error, counters);                             \
  } while (0)
  const size_t shared = 4 * sizeof(RefineShared);
  switch (scene.geometry) {
    case kGeoHalfBounds: DVS_REFINE(kGeoHalfBounds); break;
    case kGeoWatertight: DVS_REFINE(kGeoWatertight); break;
    case kGeoHalfBounds | kGeoWatertight: DVS_REFINE(kGeoHalfBounds | kGeoWatertight); break;
    default: DVS_REFINE(kGeoReference);
  }
#undef DVS_REFINE
  return cudaGetLastError();
}

cudaError_t launch_identify_exact(int n, const Cell *cells, int n_cells, double start, double end,
                                  const OpticalKnot *knots, int32_t *knot_counts, int capacity, int32_t *exact_cells,
                                  int32_t *exact_counts, int32_t *queue, int32_t *total,
                                  unsigned long long *ref_stats, cudaStream_t s) {
  identify_exact_kernel<<<blocks_of(n, 128), 128, 0, s>>>(n, cells, n_cells, start, end, knots, knot_counts, capacity,
                                                          exact_cells, exact_counts, queue, total, ref_stats);
  return cudaGetLastError();
}

cudaError_t launch_sample_exact(const SceneView &scene, const CellPose *poses, const int32_t *exact_cells,
                                const int32_t *queue, const int32_t *total, int capacity, double *exact_radiance,
                                int32_t *error, unsigned long long *counters, cudaStream_t s) {
#define DVS_EXACT(G)                                                                                       \
  sample_exact_kernel<G><<<sm_count() * 8, 128, 0, s>>>(scene, poses, exact_cells, queue, total, capacity,     \
                                                        exact_radiance, error, counters)
  switch (scene.geometry) {
    case kGeoHalfBounds: DVS_EXACT(kGeoHalfBounds); break;
    case kGeoWatertight: DVS_EXACT(kGeoWatertight); break;
    case kGeoHalfBounds | kGeoWatertight: DVS_EXACT(kGeoHalfBounds | kGeoWatertight); break;
    default: DVS_EXACT(kGeoReference);
  }
#undef DVS_EXACT
  return cudaGetLastError();
}

cudaError_t launch_integrate_knots(int n, const Cell *cells, int n_cells, double start, double end,
                                   const OpticalKnot *knots, const int32_t *knot_counts, int capacity,
                                   const int32_t *exact_cells, const double *exact_radiance,
                                   const int32_t *exact_counts, PixelParams p, PhotoParams photo, int max_events,
                                   CircuitState st, int32_t *ev_count, double *slab_t, int8_t *slab_p,
                                   int32_t *error, cudaStream_t s) {
  integrate_knots_kernel<<<blocks_of(n, 128), 128, 0, s>>>(n, cells, n_cells, start, end, knots, knot_counts,
                                                           capacity, exact_cells, exact_radiance, exact_counts, p,
                                                           photo, max_events, st, ev_count, slab_t, slab_p, error);
  return cudaGetLastError();
}

cudaError_t launch_compact_fallback(int n, const int32_t *knot_counts, int32_t *list, int32_t *total,
                                    cudaStream_t s) {
  compact_fallback_kernel<<<blocks_of(n, 128), 128, 0, s>>>(n, knot_counts, list, total);
  return cudaGetLastError();
}

cudaError_t launch_capture_probes(int n_probes, const int32_t *probe_ranks, const double *receptor_log,
                                  double *probe_state, cudaStream_t s) {
  capture_probes_kernel<<<blocks_of(n_probes, 128), 128, 0, s>>>(n_probes, probe_ranks, receptor_log, probe_state);
  return cudaGetLastError();
}

cudaError_t launch_advance_probes(int n_probes, const int32_t *probe_ranks, const Cell *cells, int c0, int nc,
                                  const double *light, const OpticalKnot *knots, const int32_t *knot_counts,
                                  int capacity, double start, double end, PhotoParams photo, double charge,
                                  double *probe_state, cudaStream_t s) {
  advance_probes_kernel<<<blocks_of(n_probes, 128), 128, 0, s>>>(n_probes, probe_ranks, cells, c0, nc, light, knots,
                                                                 knot_counts, capacity, start, end, photo, charge,
                                                                 probe_state);
  return cudaGetLastError();
}

}  // namespace dvsgb
