// A CUDA runtime without a GPU, for checks of the library's host code
// (tests/cuda/host_check.cpp): device memory is host memory that remembers its device,
// copies happen at once, streams and events remember the device they were made on,
// and the kernels write recognisable results. What CUDA would refuse or fault on
// (another device's stream, event or memory) is refused and counted.
#pragma once

#include <cstddef>
#include <cstdint>
#include <functional>
#include <vector>

#include "optx_engine.hpp"

namespace fake {

extern int devices;                 // cudaGetDeviceCount
extern thread_local int current;    // the calling thread's current device
extern bool frees_fail;             // cudaFree and friends fail, as after a device reset
extern int faults;                  // launches given another device's memory
extern int mallocs, instantiations; // calls so far
extern int history_block;           // threads per block of the last history_tally_kernel
size_t device_bytes();              // device memory allocated now
bool stale_error();                 // what the next cudaGetLastError would return is an error

extern std::function<void()> on_shares;  // called by each shares launch before it writes

// Photon `id` in the records that the fake kernels write.
inline uint8_t fate(uint64_t id) { return static_cast<uint8_t>(id % 5u); }
inline uint32_t word(uint64_t id) { return static_cast<uint32_t>(id * 2654435761u); }

// Every engine run so far: what its wave kernel was launched with.
struct Run {
  optx::WaveArgs args;
  optx::DevParams p0;
};
extern std::vector<Run> runs;

}  // namespace fake
