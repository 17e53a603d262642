// fake_cudart.h -- what a test sees of the stand-in runtime (fake_cudart.cpp)
#pragma once
#include <cuda_runtime.h>

#include <functional>
#include <map>
#include <string>

namespace fake {
extern size_t limit, used, largest;  // device memory: most that may be in use, in use, largest block so far
// called for every kernel launch with the kernel's (mangled) name and its arguments
extern std::function<void(const std::string &, void **)> on_launch;
extern std::map<std::string, int> launches;  // by name; "?" for graphs
extern thread_local unsigned grid;           // blocks of the launch that the hook sees
extern int pinned;                           // pinned allocations so far
extern int device, sms[2];                   // current device, multiprocessors of each
}  // namespace fake
