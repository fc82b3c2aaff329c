// ice_tune.h -- the flux kernel's schedule per closure (ice_sweep.cuh), set by hand from the passes below on one
// B200: one row serves the three closures. The tuner (ice_b200/tune.py) rewrites it; the library reads it at build time.
//
//   kz     the longest march of a thread along y or z, in faces (shorter where the run is small: choose_march)
//   zpass  the start of a march (the slope of its first cell), in thirds of a face: the larger, the longer
//          the marches, of a run of more threads than the GPU holds (below that every march is one face)
//   wcap   the planes of a slab, whose x, y and z faces run one after the other
//
// The environment variable ICE_GPU_TUNE="kz,zpass,wcap" overrides the row of every closure (the
// tuner's sweep uses it).
//
// Measured on single cases rather than the tuner's tree (ms a pass, kz 16 / 8 / 4 at zpass 4, wcap 4): FP32 form IG
// 128 x 126 x 129 14.80 / 14.49 / 14.67, AG 96^3 10.46 / 10.33 / 10.35, three families on 8 blocks 33.6 / 32.8 / 33.0;
// FP64 IG 96 x 95 x 97 7.82 / 7.70 / 7.75. zpass 1 to 9 and wcap 2 to 32 move them by 1 % or less.
#pragma once

namespace ice {

struct TuneRow { int kz, zpass, wcap; };

// MK, IG, AG
constexpr TuneRow kTune[3] = {
    {8, 4, 4},
    {8, 4, 4},
    {8, 4, 4},
};

}  // namespace ice
