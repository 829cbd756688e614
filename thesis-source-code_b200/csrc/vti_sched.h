// How a 3D step launch is cut into work items: columns of TX x TY points and
// segments of z planes, dealt out to persistent CTAs (host only).
#pragma once

#include <algorithm>

#include "vti_internal.h"

namespace vti {

constexpr int TX = 32, TY = 16;  // points of a column in x, y

struct Sched {
  int gx, gy;  // columns in x, y
  int nz;
  int seg;     // planes per segment
  int items;   // gx * gy * ceil(nz / seg)
  int grid;    // persistent CTAs, min(items, resident slots)
};

// Segment length: the smallest modelled time, counted in plane-steps of one
// CTA, waves * (seg + restart), where a wave is one item per resident slot
// and a restart (8 queue planes read with plain loads, pipeline refill) costs
// about kRestart plane-steps. Segments of fewer than 8 planes (down to 4) only
// while all items are resident at once: there they fill slots that would idle,
// with more waves they only add restarts.
// Measured with the alternating march (nt 300..514), restart 4 -> 1: gradient
// 300x200x90 50.3 -> 46.8 ms, 251x203x150 89.4 -> 87.9, 400x400x200 and
// 128^3..208x192x128 unchanged; short segments: 110x97x83 one-call 22.7 -> 20.4 ms,
// 112x112x96 12.2 -> 11.7 ms, allowed everywhere 160x160x112 25.0 -> 25.5 ms.
// Volumes that share a launch fill the slots together, so the waves are those of
// the whole launch (whole gradients side by side, waves of each volume alone -> of
// the launch: 24 windows of 48..80 x 48..80 x 100 cells 45.9 -> 41.6 ms, 16 of 64..96 x
// 64..96 x 64 30.7 -> 29.0, six of 96..224 x 96..224 x 100 54.8 -> 53.4, 16 of 160..400 x
// 160..400 x 200, where any length does, 231 -> 234).
constexpr long long kRestart = 1;
constexpr int kSegPlanes = 8, kSegPlanesOneWave = 4;

inline long long sched_columns(const Dims3& d) {
  return (long long)((d.nx - kHalo + TX - 1) / TX) *  // x origins 0, 32, ...; updated x < nx-4
         ((d.ny - 2 * kHalo + TY - 1) / TY);
}

// Schedule of one launch over d on sm_count SMs with ctas_per_sm resident CTAs each.
// copies: the launch works on that many volume sets at once (items per copy).
// launch_planes: column-planes (columns * nz) of all volumes that share the
// launch, d among them; 0: d alone.
inline Sched plan_sched(int sm_count, const Dims3& d, int ctas_per_sm, int copies,
                        long long launch_planes) {
  Sched s{};
  s.gx = (d.nx - kHalo + TX - 1) / TX;
  s.gy = (d.ny - 2 * kHalo + TY - 1) / TY;
  s.nz = d.nz;
  const long long cols = (long long)s.gx * s.gy * copies;
  const long long slots = (long long)sm_count * ctas_per_sm;
  long long best = -1;
  for (int nseg = 1; nseg <= d.nz; ++nseg) {
    const int seg = (d.nz + nseg - 1) / nseg;
    if (nseg > 1 && seg < kSegPlanesOneWave) break;
    if (nseg > 1 && seg == (d.nz + nseg - 2) / (nseg - 1)) continue;  // same seg
    const long long items = cols * ((d.nz + seg - 1) / seg);
    if (items > (1LL << 30)) break;
    // the launch's items, every volume in segments of about seg planes
    const long long all =
        launch_planes ? (launch_planes * ((d.nz + seg - 1) / seg) + d.nz - 1) / d.nz : items;
    const long long waves = (all + slots - 1) / slots;
    if (nseg > 1 && seg < kSegPlanes && waves > 1) continue;
    const long long cost = waves * (seg + kRestart);
    if (best < 0 || cost < best) {
      best = cost;
      s.seg = seg;
      s.items = (int)(items / copies);
    }
  }
  s.grid = (int)std::min<long long>((long long)s.items * copies, slots);
  return s;
}

}  // namespace vti
