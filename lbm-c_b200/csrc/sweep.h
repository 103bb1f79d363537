// Sweeps of several time steps through the L2 cache.
//
// A step reads and writes every population once, so a domain larger than L2
// streams through HBM at every step.  In a sweep of T steps the domain is cut
// into slabs of whole planes (z in 3-D, y in 2-D) and the T steps follow one
// another slab by slab while its planes are in L2: level s (the s-th step of
// the sweep) runs one plane further back for each level, because the step of
// a plane needs the previous step on that plane and its two neighbours.
// Slab k's level s covers the planes [start(k) - s, start(k + 1) - s); the
// first slab's level s begins at plane s instead, and the planes this leaves
// out come last, past the periodic end.  In every layout a step touches only
// the slots that hold values for its own nodes, so levels on different
// planes never meet in memory.
//
// Slabs go to two streams in turn, so that one slab's blocks fill the SMs that
// the other's last blocks leave idle: level s of slab k follows level s - 1 of
// slab k (stream order) and of slab k - 1 (an event).
#pragma once

#include <algorithm>
#include <climits>

namespace lbmc {

struct SweepPlan {
  static constexpr int MAX_DEPTH = 8;
  int depth = 1;  // steps per sweep; 1: step by step
  int slab = 0;   // planes per slab
  int planes = 0;

  // The first slab has to hold a plane of every level.
  int first_slab(int levels) const { return std::max(slab, 2 * levels + 1); }
  int slabs(int levels) const {
    const int s1 = first_slab(levels);
    return planes <= s1 ? 1 : 1 + (planes - s1 + slab - 1) / slab;
  }
  int start(int k, int levels) const { return k == 0 ? 0 : first_slab(levels) + (k - 1) * slab; }
  // Planes [begin, end) of level s of slab k; planes past the last one wrap.
  int begin(int k, int s, int levels) const { return k == 0 ? s : start(k, levels) - s; }
  int end(int k, int s, int levels) const {
    return k == slabs(levels) - 1 ? planes + s : start(k + 1, levels) - s;
  }
};

// Chooses the sweep of a domain of `planes` planes of plane_bytes each, in
// storage elements of elem bytes.  Measured on a B200 (126 MB L2), us per
// step, step by step -> swept: D3Q15 MRT 256^3 FP32 326 -> 255 (65.7 GLUPS; one
// read and one write of HBM per step would allow 54), FP16 with stochastic
// rounding 262 -> 247, Smagorinsky 256^3 BF16 259 -> 230 (both with two planes
// a block; 250 and 236 with one), 160^3 FP64 181 -> 137,
// 192^3 FP32 140 -> 107, D2Q9 4096x2048 FP32 115 -> 103.
//   - Slabs of ~30 MB: 16 MB ones (256^3 FP32, 4 planes) lose to the drain
//     between launches, 47 MB ones (12 planes: 294) to evictions.
//   - Eight levels where two slabs and the planes between the first and the
//     last level stay within ~96 MB, fewer where a plane is large (four
//     levels at 256^3: 269).
//   - Smaller domains are stepped one by one.  The line for 4- and 8-byte
//     storage is 1.25 x L2: FP32 128^3 (126 MB) ran 42.4 us swept and 43.1 us
//     not, FP64 128^3 (252 MB) 68 and 92.  2-byte storage, bound by
//     instruction issue before HBM, starts to gain later: FP16 192^3 (212 MB)
//     104.4 and 103.5, 256^3 (503 MB) 250 and 262; its line is 2 x L2.
//   - Planes above plane_limit bytes (sweep_plane_limit): step by step.
inline SweepPlan plan_sweep(int planes, long long plane_bytes, int elem, long long plane_limit = LLONG_MAX) {
  constexpr long long L2 = 126ll << 20, SLAB = 30ll << 20, WINDOW = 96ll << 20;
  SweepPlan p;
  p.planes = planes;
  if (plane_bytes > plane_limit) return p;
  if (plane_bytes * planes <= (elem > 2 ? L2 + L2 / 4 : 2 * L2)) return p;
  p.slab = (int)std::max(1ll, SLAB / plane_bytes);
  const long long skew = WINDOW / plane_bytes - 2 * p.slab;
  // at least three slabs, else there is nothing to overlap
  const long long room = (planes - 2 * p.slab - 1) / 2;
  p.depth = (int)std::max(1ll, std::min<long long>(SweepPlan::MAX_DEPTH, std::min(skew, room)));
  return p;
}

// The largest plane of a domain that gains from sweeps.  3-D domains gain, or
// lose 1% at most (2-byte storage in the shift layout), up to the planes that
// leave no second level.  In 2-D a plane is a row, one step of a short slab of
// long rows is a launch of few blocks, and the step of 2-byte storage is near
// its issue limit without a sweep.  us a step of ~20 M nodes, step by step ->
// swept, by row length:
//   - FP64: 300000 tiled 456 -> 411; never slower.
//   - FP32, tiled AA or partly solid nodes: 64000 230 -> 173, 300000 233 ->
//     211, 600000 (21.6 MB) 232 -> 328; partly solid in the shift layout
//     300000 338 -> 318, 600000 337 -> 345.  Line: 12 MB.
//   - FP32 otherwise: 100000 (3.6 MB) 267 -> 261, 120000 259 -> 259, 150000
//     (5.4 MB) 266 -> 279, 600000 262 -> 321.  Line: 4 MB.
//   - 2-byte storage, tiled AA: FP16 64000 175 -> 163, 150000 (2.7 MB) 173 ->
//     176, 200000 173 -> 163, 300000 (5.4 MB) 174 -> 192.  Line: 4 MB.
//   - 2-byte storage otherwise: FP16 BGK 6000 199 -> 215, 150000 198 -> 229, MRT
//     4000 161 -> 170, forced BGK 100000 209 -> 212: none.  With Smagorinsky or
//     with partly solid nodes and a force, whose steps are longer: 4000 189 ->
//     184 and 216 -> 207, 100000 (1.8 MB) 204 -> 200 and 235 -> 227, 150000
//     (2.7 MB) 248 -> 257 and 281 -> 281.  Line: 2 MB.
inline long long sweep_plane_limit(int dim, int elem, bool tiled, bool smagorinsky, bool partly_solid, bool forcing) {
  constexpr long long MB = 1ll << 20;
  if (dim == 3 || elem == 8) return LLONG_MAX;
  if (elem == 4) return tiled || partly_solid ? 12 * MB : 4 * MB;
  if (tiled) return 4 * MB;
  return smagorinsky || (partly_solid && forcing) ? 2 * MB : 0;
}

}  // namespace lbmc
