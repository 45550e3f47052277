// Engine<float>::ensure_workspace on the CPU, with stand-ins for the library's
// allocator and error functions: the allocation number argv[1] fails.  Prints for
// two calls in a row: return code, whether zhat and slab are there, blocks held.
#include <cstdio>
#include <cstdlib>
#include <set>
#include "engine.h"

namespace ddb {
static int g_fail = 0, g_count = 0;
static std::set<void*> g_held;
cudaError_t dev_alloc(void** p, size_t) {
  *p = nullptr;
  if (++g_count == g_fail) return cudaErrorMemoryAllocation;
  *p = std::malloc(1);
  g_held.insert(*p);
  return cudaSuccess;
}
void dev_free(void* p) {
  if (p) { g_held.erase(p); std::free(p); }
}
void set_error(const char*, const char*) {}
void set_cuda_error(const char*, cudaError_t) {}
void clear_error() {}
int check_launch(const char*) { return 0; }
void raise_smem_limit(const void*) {}
bool env_flag(const char*) { return false; }
void note_launch(unsigned long long) {}
}  // namespace ddb

int main(int argc, char** argv) {
  ddb::g_fail = argc > 1 ? std::atoi(argv[1]) : 0;
  ddb::Engine<float> e;
  e.g.nx = e.g.ny = e.g.nz = 8;
  e.g.Mx = e.g.My = e.g.Mz = 16;
  e.g.nat = 512;
  e.xpipe = 1;
  e.slab_budget_elems = (size_t)1 << 28;
  for (int call = 0; call < 2; ++call) {
    const int rc = e.ensure_workspace(2);
    std::printf("%d %d %d %d %zu\n", rc, e.zhat != nullptr, e.slab != nullptr, (int)ddb::g_held.size(), e.bytes_allocated);
  }
  return 0;
}
