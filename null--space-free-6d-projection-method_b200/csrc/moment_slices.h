// How the FP64 Taylor moments cut their modes (host only).
#pragma once
#include <algorithm>

namespace fame {

// NF modes in slices of whole stages (of `stage` modes), for `tiles` CTAs per slice on `slots`
// places: whole waves, at least four stages each, at most `most` modes (a multiple of the stage),
// so that the accumulation error of a slice does not grow with the number of centers.
inline void moment_slices(long long NF, long long tiles, long long slots, long long stage, long long most, int* nslices,
                          long long* per_slice) {
  const long long waves = std::max<long long>(1, (NF * tiles + slots * most - 1) / (slots * most));
  // waves * slots / tiles rounds down: with hundreds of tiles that alone would pass `most`
  const long long want = std::max<long long>((NF + most - 1) / most, waves * slots / tiles);
  const long long per = std::max<long long>(4 * stage, (NF + want - 1) / want);
  *per_slice = (per + stage - 1) / stage * stage;
  *nslices = (int)((NF + *per_slice - 1) / *per_slice);
}

}  // namespace fame
