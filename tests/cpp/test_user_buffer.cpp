// Routes of caller's pointers (user_buffer.h) on made-up attributes: no GPU needed.
#include <cstdio>

#include "user_buffer.h"

static int bad = 0;
#define CHECK(x) \
  do { \
    if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); bad = 1; } \
  } while (0)

static cudaPointerAttributes at(cudaMemoryType t, int device) {
  cudaPointerAttributes a{};
  a.type = t;
  a.device = device;
  return a;
}

int main() {
  using namespace opfc;
  for (int dev = 0; dev < 8; ++dev) {
    CHECK(own_device_memory(at(cudaMemoryTypeDevice, dev), dev));
    CHECK(!own_device_memory(at(cudaMemoryTypeDevice, dev + 1), dev));
    CHECK(!own_device_memory(at(cudaMemoryTypeManaged, dev), dev));
    CHECK(!own_device_memory(at(cudaMemoryTypeHost, dev), dev));
    CHECK(!own_device_memory(at(cudaMemoryTypeUnregistered, dev), dev));
    CHECK(pinned_host_memory(at(cudaMemoryTypeHost, dev)));
    CHECK(!pinned_host_memory(at(cudaMemoryTypeDevice, dev)));
    CHECK(!pinned_host_memory(at(cudaMemoryTypeManaged, dev)));
    CHECK(!pinned_host_memory(at(cudaMemoryTypeUnregistered, dev)));
  }
  return bad;
}
