// Prints, for a sweep of traces and every tuning of the sub-rays per lane, the
// calls that break a rule of the traces' shapes (batch.cu, kernels.cu).
#include <cstdio>

#include "kernels.h"

using namespace dvsgb;

int main() {
  long traces = 0, beams = 0, broken = 0;
  for (int samples : {1, 2, 3, 4, 5, 6, 8, 16})
    for (int geometry : {0, 1, 2, 3})
      for (int n_pix : {1, 31, 300, 3072, 32768, 89960, 921600})
        for (int nc : {1, 3, 7, 8, 9, 33, 64, 640})
          for (int cw_log2 = 0; cw_log2 <= 5; ++cw_log2)
            for (bool scattered : {false, true}) {
              SceneView v{};
              v.samples = samples;
              v.geometry = geometry;
              const int ss2 = samples * samples;
              const bool beam = trace_item_shape(n_pix, nc, cw_log2, ss2, 1, scattered).beam;
              beams += beam;
              int walk[5] = {};
              for (int rays : {0, 1, 2, 4}) {
                v.rays = rays;
                const int got = trace_rays(v, n_pix, nc, cw_log2, scattered);
                const ItemShape shape = trace_item_shape(n_pix, nc, cw_log2, ss2, got, scattered);
                ++traces;
                walk[rays] = got;
                // where one ray per lane shares a walk, every tuning takes it; no other ray count ever does
                const bool ok = ss2 % got == 0 && (beam ? got == 1 && shape.beam : !shape.beam);
                if (!ok) ++broken;
              }
              // without one the tuning holds, as far as the sub-rays divide; automatically two
              if (!beam && (walk[0] != walk[2] || walk[1] != 1 || walk[2] != (ss2 % 2 ? 1 : 2) ||
                            walk[4] != (ss2 % 4 == 0 && geometry == 0 ? 4 : walk[2])))
                ++broken;
            }
  // items of a trace by poses fill their packets where there are items enough for the GPU; scattered pixels, whose beam
  // would be too wide, hold just one packet and share none
  long poses = 0;
  for (int samples : {1, 2, 3, 4, 5, 6, 8, 16})
    for (int n_pix : {1, 31, 1024, 89960, 921600})
      for (int nc = 1; nc < 8; ++nc)
        for (bool scattered : {false, true}) {
          SceneView v{};
          v.samples = samples;
          if (!trace_by_pose(v, n_pix, nc)) continue;
          ++poses;
          const PoseShape s = pose_item_shape(n_pix, nc, samples * samples, scattered);
          const int per_packet = 32 >> s.lanes_log2;
          const bool many = (long long)n_pix * nc >= 32 * 4864;
          if (s.pixels < 1 || s.pixels > 32 || (many && s.pixels < per_packet) ||
              (scattered && (s.pixels > per_packet || (s.beam && s.pixels > 1))))
            ++broken;
        }
  if (!poses) ++broken;
  std::printf("traces %ld\nbeams %ld\nbroken %ld\n", traces, beams, broken);
  return 0;
}
