// pt_forms.h — up to which size an image, a batch or a frame of the cached renderer runs in the kernel of pt_paths.h
// instead of the wavefront (`lanes`: the kernel's resident threads).
//
// The kernel gains where most paths of an image end early: the wavefront's queues then soon are too short to fill
// the GPU, while its lanes take the next sample.  Where paths go on for many bounces (inside a room) the queues
// stay long, and kernels that only walk or only shade keep 32 lanes busy where the one kernel shades about half
// of a warp at a time.  Which of the two a view is, is looked at before the first call: 1,024 camera paths, two
// diffuse bounces each (probe_path in pt_paths.h, some 0.1 ms, only for images of a size that the answer matters for).
//
// Measured, time of the wavefront over the time of the kernel (five blocks per SM, 94,720 lanes), on open scenes
// (displaced spheres on a floor):
//   pixels per lane           6.1        15      22      30      39
//   10,000 triangles, 1 spp   1.8        -       1.4     1.3     1.2       16 spp 1.8, -, 1.3, 1.2, 1.06
//   200,000, 1 spp            -          1.3     1.16    1.07    1.0       16 spp -, 1.4, 1.25, 1.14, 1.06
//   1M, 1 spp                 1.4        1.1     1.03    0.93    0.88      4 spp 1.6, 1.24, 1.10, 1.03, 0.96
//   1M, 1 spp, limit 2        1.12       0.91    0.86    -       -         4 spp 1.6, 1.17, 1.04
//   65,000, 1 spp, limit 2    -          1.17    1.04    -       0.96      4 spp -, 1.4, 1.2, -, 1.03
// and inside a room (the Cornell box with every triangle split; bounce limit 8, 1 and 16 spp):
//   pixels per lane           2.4          6.1          22
//   1,280 triangles           0.85 0.99    0.71 0.74    0.58 0.62
//   20,480                    1.16 1.68    0.83 0.95    0.62 0.67
//   327,680                   1.8  3.7     1.3  1.9     0.74 0.86
// A room that has lost four to eight of its ten wall triangles (0.67 to 0.98 at 4 to 22 pixels per lane) is still a room.
#pragma once

#include <cmath>
#include <cstddef>
#include <cstdint>

namespace ptb {

constexpr int kProbeSide = 32;                               // the probe's image
constexpr int kProbePaths = kProbeSide * kProbeSide;
// Whether the paths of a probe go on: five surfaces met for four paths (a path meets two at most).  The open scenes
// above meet 0.8 to 1.03 a path, the rooms 1.45 to 2.
inline bool paths_go_on(uint32_t met) { return 4 * met >= 5 * uint32_t(kProbePaths); }

// Most pixels per lane of a view whose paths go on: the longer the walks, the longer the wavefront waits for its
// slowest rays.
inline double most_pixels_going_on(size_t primitives) { return 0.35 * std::pow(double(primitives), 0.25); }

// Most pixels per lane of an open view in a call of `bounces` = samples x bounce limit: the last paths of a call are a
// smaller part of a long one.  The wavefront's walk kernels hold more warps, which counts on trees out of the L1's reach.
// Past the L2 (2.6M overlapping triangles, 8 spp and more 1.29 at 6.1, 1.12 at 9.7, 0.92 at 22; 1 spp of limit 2 0.82 at 6.1).
inline double most_pixels_open(size_t walked_bytes, int64_t bounces) {
    if (walked_bytes <= (size_t(8) << 20)) return bounces < 4 ? 25 : 40;
    if (walked_bytes > (size_t(100) << 20)) return bounces < 8 ? 5 : 14;
    return bounces < 8 ? 12 : bounces < 32 ? 25 : bounces < 128 ? 32 : 40;
}

// Up to how many pixels per lane an image runs in the tail kernel alone, whose two lanes per path walk extension and
// shadow rays side by side.  Where walks are short a call of several samples gains by it for longer (tail kernel alone
// over the kernel of pt_paths.h, 4 and 16 spp at 2.0, 2.7 and 4.1 pixels per lane: 400 triangles 0.81 0.69, 0.88 0.72, 1.08
// 0.83; 10,000 0.88 0.84, 0.97 0.86, 1.03 1.02; 65,000 0.89 0.86, 0.89 0.89, 1.16 1.19; 200,000 0.97 0.94, 1.07 1.00, 1.26
// 1.20; 1M 1.15 1.11, 1.35 1.37, 1.56 1.71; of one sample 1.02 to 1.27 at 2.0 on all but 200,000 triangles).
inline double most_pixels_alone(bool go_on, size_t walked_bytes, int64_t samples) {
    return !go_on && walked_bytes <= (size_t(8) << 20) && samples >= 4 ? 3 : 2;
}

// Most pixels per lane of an image.
inline double most_pixels(bool go_on, size_t primitives, size_t walked_bytes, int64_t bounces) {
    return go_on ? most_pixels_going_on(primitives) : most_pixels_open(walked_bytes, bounces);
}

// A batch mixes both.  Open jobs fill the lanes that the others' paths leave idle (two Cornell boxes among six jobs,
// pixels per lane in all, of the boxes and gain: 7.5 2.4 1.18; 10 3.2 1.09; 12.7 4.1 1.0; 15 4.9 0.94; 24 7.6 0.82).  Open
// jobs alone, 8 spp: 10,000 triangles 1.06 at 31 pixels per lane, 65,000 1.03, 1M 1.04 at 21 and 0.92 at 31.
inline bool batch_in_one(double open_pixels, double going_on_pixels, double most_going_on, size_t walked_bytes, double lanes) {
    const double open = open_pixels / lanes, going_on = going_on_pixels / lanes;
    return open + going_on <= (walked_bytes <= (size_t(8) << 20) ? 30 : walked_bytes <= (size_t(100) << 20) ? 22 : 6) &&
           (going_on_pixels <= 0 || going_on <= (most_going_on > 1 ? most_going_on : 1) + open / 3);
}

// The cached renderer's paths end at their first query (without its cache it is the plain renderer), so rooms gain for
// longer (pixels per lane, samples x limit 48; wavefront over kernel): 1,280 triangles 0.98 at 6.1, 0.70 at 22; 20,480 1.36, 0.84; 327,680 2.25, 1.33.
// Open views: 20 pixels per lane, 28 when the bounces of a frame are many (65,000 triangles at 15 and 22: 1.27 and
// 1.10; 1M 1.33 and 1.15; of one sample 1.13 and 1.04 at 15, none measured above); half of that past the L2 (2.6M, one
// sample 1.03 at 6.1 and 0.90 at 15, four 1.11 at 9.7 and 0.94 at 15).
inline double most_pixels_cached(bool go_on, size_t primitives, size_t walked_bytes, int64_t bounces) {
    const double most = (bounces >= 24 ? 28 : 20) / (walked_bytes <= (size_t(100) << 20) ? 1.0 : 2.0);
    const double room = 1.1 * std::pow(double(primitives), 0.25);
    return go_on && room < most ? room : most;
}

} // namespace ptb
