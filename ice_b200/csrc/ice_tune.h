// ice_tune.h -- the flux kernel's schedule per closure (ice_sweep.cuh), as the tuner (ice_b200/tune.py) chose
// it by timing the stage on one B200. Rewritten by the tuner; the library reads it at build time.
//
//   kz     the longest march of a thread along y or z, in faces (shorter where the run is small: choose_march)
//   zpass  the start of a march (the slope of its first cell), in thirds of a face: the larger, the longer
//          the marches a small run takes
//   wcap   the planes of a slab, whose x, y and z faces run one after the other
//
// The environment variable ICE_GPU_TUNE="kz,zpass,wcap" overrides the row of every closure (the
// tuner's sweep uses it).
#pragma once

namespace ice {

struct TuneRow { int kz, zpass, wcap; };

// MK, IG, AG
constexpr TuneRow kTune[3] = {
    {16, 4, 8},
    {16, 4, 8},
    {16, 4, 8},
};

}  // namespace ice
