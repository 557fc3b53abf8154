// What the stub of the CUDA runtime knows of the library's kernels (decode.cu).
#pragma once
#include <functional>
#include <string>
#include <vector>

struct StubLaunch {
  std::vector<const void*> objects;                // working counters that the launch changes
  bool null_argument = false;                      // a buffer that the kernel uses is null
  std::function<void(bool)> counts = [](bool) {};  // leaves the frame's counts on the host: an overflow, or none
  // logged: view_proj[12] of the scenes drawn; of reyes_split the places on a frontier and for leaves
  std::function<std::vector<float>()> cameras = [] { return std::vector<float>(); };
};

// What the next Reyes frame reports (stub_patches)
extern unsigned stub_frontier, stub_leaves;

// "raster_setup", ... from the mangled name
std::string stub_kernel_name(const char* mangled);
// A launch's arguments, copied
StubLaunch stub_decode(const char* name, void** args);
