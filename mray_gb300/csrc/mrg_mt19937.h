// mrg_mt19937.h -- outputs of std::mt19937 made on the device.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace mrg {

// out[i] = output `first` + i of std::mt19937(seed), i < count; with `pcg` the
// PermutedCG32 state it seeds (PermutedCG32::GenerateState, Source/Tracer/
// Random.h): (x + increment) * multiplier + increment.
cudaError_t mt19937_outputs(uint32_t seed, uint64_t first, uint32_t count, bool pcg, uint32_t* out, cudaStream_t st);

} // namespace mrg
