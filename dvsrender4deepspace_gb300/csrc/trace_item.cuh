// Per-item device bodies of the trace and circuit launches, shared by the
// one-sensor kernels (kernels.cu) and the multi-sensor batch kernels
// (batch.cu).  Included after device_optics.cuh and device_circuit.cuh.
#pragma once
#include "device_circuit.cuh"
#include "device_optics.cuh"

namespace dvsgb {
namespace {

constexpr int kWarpsPerBlock = 4;  // all ray kernels launch 128 threads
// Resident blocks per SM the trace kernel is compiled for: 5 blocks of 128
// threads cap it at 96 registers (20 warps per SM), the fastest measured
// balance of latency hiding against register spills.
#ifndef DVS_TRACE_MIN_BLOCKS
#define DVS_TRACE_MIN_BLOCKS 5
#endif
constexpr int kSubrayTable = 256;  // sub-rays per pixel with a shared sub-ray table (ss <= 16)

// A warp's shared memory in the trace kernels: the traversal stack and the
// sub-ray table (and, in kernels with beams, a Beam beside it).
struct TraceShared {
  int code[kStackSlots];
  float t[kStackSlots];
  SubraySample subrays[kSubrayTable];
};

// Element o of a radiance chunk: double, or float when the chunk feeds an
// FP32 circuit (which uses the value as a float: the same bits, half the bytes).
__device__ __forceinline__ void store_radiance(const SceneView &S, double *chunk, size_t o, double value) {
  if (S.radiance_f32) reinterpret_cast<float *>(chunk)[o] = (float)value;
  else chunk[o] = value;
}
// Several sub-rays per lane (SceneView::rays: 1, 2 or 4, when the pixel's
// sub-ray count is a multiple): the kernels with more ray state per lane are
// compiled for fewer resident blocks (more registers).
#ifndef DVS_TRACE_PAIR_MIN_BLOCKS
#define DVS_TRACE_PAIR_MIN_BLOCKS 4
#endif
#ifndef DVS_TRACE_BEAM_MIN_BLOCKS
#define DVS_TRACE_BEAM_MIN_BLOCKS 5
#endif
#ifndef DVS_TRACE_QUAD_MIN_BLOCKS
#define DVS_TRACE_QUAD_MIN_BLOCKS 3
#endif

// The ranges of every ray of an item -- its pixel sets [s0, s1) at its cell
// groups [g0, g1) -- into the beam, and its leaf list.  Directions: the
// corner sub-rays of each pixel at each cell.  Between the corners a
// normalized direction bends by at most about its extent squared; the margin
// covers that, and each packet checks its rays against the range.
template <int kGeo>
__device__ __forceinline__ BeamLists begin_beam(const SceneView &S, int n_pix, const int32_t *rank_list,
                                                const CellPose *poses, int c0, int nc, int cw_log2, int s0, int s1,
                                                int g0, int g1, Beam &B, int *stack) {
  const int lane = threadIdx.x & 31, cw = 1 << cw_log2, ppw = 32 >> cw_log2, last = S.samples - 1;
  const float inf = kInf();
  float3 olo = f3(inf, inf, inf), ohi = -olo, dlo = olo, dhi = -olo, llo = olo, lhi = -olo;
  for (int s = s0; s < s1; ++s) {
    const int rank = s * ppw + (lane >> cw_log2);
    const int pixel = rank < n_pix ? __ldg(S.pixel_of_rank + (rank_list ? rank_list[rank] : rank)) : 0;
    const int px_i = pixel % S.width, py_i = pixel / S.width;
    const float x0 = subray_x(S, px_i, 0), x1 = subray_x(S, px_i, last);
    const float y0 = subray_y(S, py_i, 0), y1 = subray_y(S, py_i, last);
    for (int g = g0; g < g1; ++g) {
      const int cell = g * cw + (lane & (cw - 1));
      if (rank >= n_pix || cell >= nc) continue;
      const CellPose pose = poses[c0 + cell];
      const float3 o = f3(pose.px, pose.py, pose.pz), l = inverse_direction(f3(pose.lx, pose.ly, pose.lz));
      olo = min3(olo, o);
      ohi = max3(ohi, o);
      llo = min3(llo, l);
      lhi = max3(lhi, l);
      for (int k = 0; k < (last ? 4 : 1); ++k) {
        const float3 d = unit(rotate_ray(pose, f3(k & 1 ? x1 : x0, -(k & 2 ? y1 : y0), -1)));
        dlo = min3(dlo, d);
        dhi = max3(dhi, d);
      }
    }
  }
  return close_beam<kGeo>(S, olo, ohi, dlo, dhi, llo, lhi, 0.0f, B, stack);
}

// A sample of an item without lists (under one in a hundred on the terrains measured), or one whose rays left the
// beam, out of line: two sub-rays per lane where their count is even, as a launch without beams.
// (The pose by its address in global memory: a reference to the caller's would hold it in local memory.)
template <int kMode, int kGeo>
__device__ __noinline__ PixelSample sample_without_beam(const SceneView &S, int pixel, bool active,
                                                        const CellPose *pose_at, TraceShared &sh,
                                                        const SubraySample *subrays) {
  const CellPose pose = *pose_at;
  if (S.samples % 2 == 0)
    return sample_pixel_group<kMode, 2, kGeo, false>(S, pixel, active, pose, sh.code, sh.t, subrays, nullptr, nullptr);
  return sample_pixel_group<kMode, 1, kGeo, false>(S, pixel, active, pose, sh.code, sh.t, subrays, nullptr, nullptr);
}

// One warp's item of a trace launch: shape.sets pixel sets (32/CW
// Morton-adjacent pixels each) x shape.groups cell groups (CW consecutive
// cells each) of one sensor, a packet of 32 x kRays rays at a time.  Called by
// trace_cells_kernel (one item per warp) and by the batch's persistent kernel
// (items pulled from a work counter).
template <int kMode, int kRays, int kGeo, bool kBeam>
__device__ __forceinline__ void trace_cells_item(const SceneView &S, int n_pix, const int32_t *rank_list,
                                                 const CellPose *poses, int c0, int nc, ItemShape shape,
                                                 double *radiance, float *depth_out, unsigned long long *counters,
                                                 long long item, TraceShared &sh, Beam &beam) {
  // n_pix pixels: all Morton ranks, or the ranks listed in rank_list
  const int lane = threadIdx.x & 31, cw_log2 = shape.cw_log2;
  const int cw = 1 << cw_log2, ppw = 32 >> cw_log2;
  const int n_groups = (nc + cw - 1) >> cw_log2, n_sets = (n_pix + ppw - 1) / ppw;
  const int per_set = (n_groups + shape.groups - 1) / shape.groups;
  const long long first_set = item / per_set * shape.sets;
  if (first_set >= n_sets) return;  // warp-uniform
  const int s0 = (int)first_set, s1 = min(n_sets, s0 + shape.sets);
  const int g0 = (int)(item % per_set) * shape.groups, g1 = min(n_groups, g0 + shape.groups);
  const int ss2 = S.samples * S.samples;
  BeamLists lists{kNoList, kNoList, 0};
  if (kBeam && shape.beam)
    lists = begin_beam<kGeo>(S, n_pix, rank_list, poses, c0, nc, cw_log2, s0, s1, g0, g1, beam, sh.code);
  unsigned primary = 0, shadow = 0;
  for (int set = s0; set < s1; ++set) {
    const int rank = set * ppw + (lane >> cw_log2);
    const int pixel = rank < n_pix ? __ldg(S.pixel_of_rank + (rank_list ? rank_list[rank] : rank)) : 0;
    // the set's ppw pixels: their sub-rays' coordinates and FP64 cos^4 once per
    // set (entry p * ss2 + j: sub-ray j of the pixel in lanes p * cw ...)
    const int table = ppw * ss2;
    const bool shared_subrays = table <= kSubrayTable;
    if (shared_subrays) {
      for (int q0 = 0; q0 < table; q0 += 32) {  // warp-uniform: every lane takes part in the shuffle
        const int q = q0 + lane, p = min(q / ss2, ppw - 1);
        const int pix = __shfl_sync(kFull, pixel, p << cw_log2);
        if (q < table) {
          const int j = q - p * ss2;
          const float x = subray_x(S, pix % S.width, j % S.samples), y = subray_y(S, pix / S.width, j / S.samples);
          sh.subrays[q] = SubraySample{cos4_of(x, y), x, y};
        }
      }
      __syncwarp();
    }
    const SubraySample *mine = shared_subrays ? sh.subrays + (lane >> cw_log2) * ss2 : nullptr;
    for (int g = g0; g < g1; ++g) {
      const int cell = g * cw + (lane & (cw - 1));
      const bool active = rank < n_pix && cell < nc;
      const CellPose *at = poses + c0 + (active ? cell : 0);
      const CellPose pose = *at;
      PixelSample s;
      bool by_list = !kBeam || lists.shadow >= 0;
      if (by_list) {
        s = sample_pixel_group<kMode, kRays, kGeo, kBeam>(S, pixel, active, pose, sh.code, sh.t, mine, &beam, &lists);
        by_list = !s.redo;
      }
      if (kBeam && !by_list) s = sample_without_beam<kMode, kGeo>(S, pixel, active, at, sh, mine);
      if (active) {
        const size_t o = (size_t)cell * n_pix + rank;
        store_radiance(S, radiance, o, s.valid ? s.radiance : __longlong_as_double(0x7ff8000000000000ll));
        if (depth_out) depth_out[o] = s.depth;
      }
      primary += s.primary;
      shadow += s.shadow;
    }
    __syncwarp();  // the table is rewritten for the next set, the lists for the warp's next item
  }
  const unsigned prim = warp_sum(primary), shad = warp_sum(shadow);
  if (lane == 0 && counters) {
    atomicAdd(counters + kCntPrimary, (unsigned long long)prim);
    atomicAdd(counters + kCntShadow, (unsigned long long)shad);
  }
}

// Few poses per pixel (camera frames, the initial pose, short exposures, the
// adaptive probes): a warp's item is several pixels at one pose, its packets 32
// sub-rays of one pixel, or of as many pixels as they fill, through the item's
// beam.  After each run of sub-rays the lanes, one per pixel, add its terms in
// sub-ray order: the FP64 sums of the serial loop, for all the item's
// pixels at once.  (One lane summing its pixel's 64 terms of a packet through shuffles, and no beam, took
// 69 ms for a 1280x720 frame with 256 sub-rays, the FP64 pipe busy with one lane's sums.)
constexpr int kPoseTerms = 288;  // pixels x (sub-rays of a run + 1)
struct PoseShared {
  int code[kStackSlots];
  float t[kStackSlots];
  Beam beam;
  double term[kPoseTerms];
  float hit_t[kPoseTerms];
};
template <int kMode, int kGeo>
__device__ __forceinline__ void trace_pose_item(const SceneView &S, int n_pix, const int32_t *rank_list,
                                                const CellPose &pose, int cell, PoseShape shape, double *radiance,
                                                float *depth_out, unsigned long long *counters, int first,
                                                PoseShared &sh) {
  const int lane = threadIdx.x & 31, count = min(shape.pixels, n_pix - first);
  const int run = 1 << shape.lanes_log2, per_packet = 32 >> shape.lanes_log2;
  const int sub = lane & (run - 1), ss2 = S.samples * S.samples;
  int pixel = 0;  // of lane i: the item's pixel i
  if (lane < count) pixel = __ldg(S.pixel_of_rank + (rank_list ? rank_list[first + lane] : first + lane));
  BeamLists lists{kNoList, kNoList, 0};
  if (shape.beam) {
    const float3 o = f3(pose.px, pose.py, pose.pz), l = inverse_direction(f3(pose.lx, pose.ly, pose.lz));
    float3 dlo = f3(kInf(), kInf(), kInf()), dhi = -dlo;
    if (lane < count) {
      const int px_i = pixel % S.width, py_i = pixel / S.width, last = S.samples - 1;
      for (int k = 0; k < (last ? 4 : 1); ++k) {
        const float3 d = unit(rotate_ray(pose, f3(subray_x(S, px_i, k & 1 ? last : 0),
                                                  -subray_y(S, py_i, k & 2 ? last : 0), -1)));
        dlo = min3(dlo, d);
        dhi = max3(dhi, d);
      }
    }
    lists = close_beam<kGeo>(S, o, o, dlo, dhi, l, l, 0.0f, sh.beam, sh.code);
  }
  double sum = 0, depth = 0;
  int valid_depth = 0;
  unsigned primary = 0, shadow = 0;
  for (int r0 = 0; r0 < ss2; r0 += run) {
    for (int s0 = 0; s0 < count; s0 += per_packet) {
      const int p = s0 + (lane >> shape.lanes_log2), r = r0 + sub;
      const int pix = __shfl_sync(kFull, pixel, min(p, 31));
      const bool live = p < count && r < ss2;
      const int rr = live ? r : 0;
      const RaySample s = sample_ray<kGeo, false>(S, subray_x(S, pix % S.width, rr % S.samples),
                                                  subray_y(S, pix / S.width, rr / S.samples), pose, live, sh.code,
                                                  sh.t, sh.beam, lists);
      if (live) {
        const int at = p * (run + 1) + sub;
        sh.term[at] = s.overflow ? __longlong_as_double(0x7ff8000000000000ll) : s.term;
        if (kMode != kRadiance) sh.hit_t[at] = s.hit ? s.t : -1.0f;
      }
      primary += live ? 1u : 0u;
      shadow += s.lit ? 1u : 0u;
    }
    __syncwarp();
    if (lane < count) {
      const int m = min(run, ss2 - r0), at = lane * (run + 1);
      for (int i = 0; i < m; ++i) {
        sum += sh.term[at + i];
        if (kMode != kRadiance && sh.hit_t[at + i] >= 0.0f) {
          depth += sh.hit_t[at + i];
          ++valid_depth;
        }
      }
    }
    __syncwarp();
  }
  if (lane < count) {
    const size_t o = (size_t)cell * n_pix + first + lane;
    store_radiance(S, radiance, o, sum / ss2);
    if (kMode != kRadiance) depth_out[o] = valid_depth ? float(depth / valid_depth) : -1.0f;
  }
  const unsigned prim = warp_sum(primary), shad = warp_sum(shadow);
  if (lane == 0 && counters) {
    atomicAdd(counters + kCntPrimary, (unsigned long long)prim);
    atomicAdd(counters + kCntShadow, (unsigned long long)shad);
  }
}

// One pixel of a circuit launch (generate_pixels' circuit half,
// event_sensor.cu:35-50, over one cell chunk): thread r of the launch
// integrates rank rank_list[r] (or r) from radiance row r.  Called by
// circuit_kernel and by the batch's multi-sensor circuit kernel.
template <bool kF32, bool kPhilox>
__device__ __forceinline__ void circuit_rank(int r, int n, const int32_t *rank_list, const Cell *cells, int c0, int nc,
                                             const double *radiance, const PixelParams &p, const PhotoParams &photo,
                                             int max_events, const CircuitState &st, int32_t *ev_count,
                                             double *slab_t, int8_t *slab_p, int32_t *error,
                                             unsigned long long *counters) {
  const int k = rank_list ? rank_list[r] : r;
  int cnt = ev_count[k];
  if (cnt < 0) return;  // failed earlier in this batch
  const bool need_rng = !kPhilox && (photo.shot_noise || p.reset_noise_std > 0);
  curandStateXORWOW_t rng;
  if (need_rng) rng = st.rng[k];
  double *my_t = slab_t + (size_t)k * max_events;
  int8_t *my_p = slab_p + (size_t)k * max_events;
  int failed = 0;
  if (!kF32) {
    CircuitRun run = circuit_begin(st, k, p);
    for (int c = 0; c < nc; ++c) {
      const Cell cell = cells[c0 + c];
      const double rad = radiance[(size_t)c * n + r];
      if (!finite_bits(rad)) { failed = kErrOptical; break; }
      double rate = rad * photo.electrons_per_radiance + photo.dark_electrons;
      if (photo.shot_noise) rate = quotient(poisson_electrons(rng, rate * cell.len), cell.len, cell.inv_len);
      const int emitted = circuit_cell(run, p, rate, cell, my_t + cnt, my_p + cnt, max_events - cnt, rng);
      if (emitted == -1) { failed = kErrCapacity; break; }
      if (emitted == -2) { failed = kErrStalled; break; }
      cnt += emitted;
    }
    circuit_end(run, st, k);
  } else {
    // precision mode: the state is held in FP32 registers for the chunk
    PixelRegsF s{(float)st.receptor_log[k], (float)st.reference_log[k], st.refractory_until[k],
                 (float)st.threshold_pos[k], (float)st.threshold_neg[k], st.reset_pending[k] != 0, true};
    const int pixel = kPhilox ? st.pixel[k] : 0;
    const float e_rad = (float)photo.electrons_per_radiance, dark = (float)photo.dark_electrons;
    const PixelParamsF pf = pixel_params_f32(p);
    const float *chunk_f = photo.chunk_f32 ? reinterpret_cast<const float *>(radiance) : nullptr;
    for (int c = 0; c < nc; ++c) {
      const Cell cell = cells[c0 + c];
      const size_t o = (size_t)c * n + r;
      const float rad = chunk_f ? chunk_f[o] : (float)radiance[o];
      if (!isfinite(rad)) { failed = kErrOptical; break; }
      float rate = photo.drawn ? rad : rad * e_rad + dark;
      const float dt = cell.dt;
      int emitted;
      if (kPhilox) {
        curandStatePhilox4_32_10_t ph{};
        if (!photo.drawn) {  // drawn: nothing more is taken from the stream
          ph = philox_at(photo.seed, pixel, cell.t0);
          if (photo.shot_noise) rate = poisson_electrons_philox(ph, rate * dt) / dt;
        }
        emitted = advance_pixel_f32(s, p, pf, rate, cell.t0, dt, my_t + cnt, my_p + cnt, max_events - cnt, ph);
      } else {
        if (photo.shot_noise) rate = (float)poisson_electrons(rng, (double)(rate * dt)) / dt;
        emitted = advance_pixel_f32(s, p, pf, rate, cell.t0, dt, my_t + cnt, my_p + cnt, max_events - cnt, rng);
      }
      if (emitted == -1) { failed = kErrCapacity; break; }
      if (emitted == -2) { failed = kErrStalled; break; }
      cnt += emitted;
    }
    st.receptor_log[k] = s.receptor_log;
    st.reference_log[k] = s.reference_log;
    st.refractory_until[k] = s.refractory_until;
    st.reset_pending[k] = s.reset_pending ? 1 : 0;
  }
  if (need_rng) st.rng[k] = rng;
  if (failed) {
    atomicOr(error, failed);
    ev_count[k] = -1;
  } else {
    ev_count[k] = cnt;
  }
  if (counters && (threadIdx.x & 31) == 0) {
    const int active = min(32, n - (r & ~31));
    atomicAdd(counters + kCntCells, (unsigned long long)active * (unsigned long long)nc);
  }
}

}  // namespace
}  // namespace dvsgb
