// A CUDA runtime without a GPU, for tests of the library's host paths: device
// memory is host memory, kernels do not run, and what the host side asked for
// is on record.  Linked with the library's own objects in place of cudart.
#pragma once

#include <cstddef>
#include <functional>
#include <map>
#include <set>
#include <string>
#include <utility>
#include <vector>

namespace fake {

struct State {
  int device = 0;
  int sms = 152;
  std::map<std::string, std::pair<unsigned, unsigned>> grids;  // of each kernel's last launch
  // copies from pageable memory run when their stream is waited for, as they
  // may where the device reads pageable memory directly
  bool defer_copies = false;
  int fail_mallocs = 0;          // the next cudaMalloc calls that fail
  size_t memory = (size_t)-1;    // device bytes in all; cudaMalloc fails past them
  size_t in_use = 0;
  bool capturing = false;        // every stream but the library's own is being captured: a wait is an error
  int recorded = 0;              // memsets that a capture only records
  int waits = 0;                 // cudaStreamSynchronize calls
  // dynamic shared memory opted into, per device and kernel name
  std::map<std::pair<int, std::string>, int> opted_in;
  // (kernel, dynamic shared bytes) launched without the opt-in it needs
  std::vector<std::string> refused;
  std::map<std::string, int> launches;
  std::function<void(const std::string& kernel, void** args)> on_launch;
  std::function<void()> on_wait;  // after a wait for a stream
};

State& state();
int device_of(const void* p);  // the device whose allocation holds p, or -1
size_t kept_on(int device);    // device bytes allocated on it

}  // namespace fake
