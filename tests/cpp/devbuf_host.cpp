// Device buffers on a host-side allocator with a size limit: what a refused
// growth leaves behind, and how much the outgrown blocks hold together.
#include <cstdio>
#include <cstdlib>
#include <map>

#include "../../pwdft_develop_b200/csrc/devbuf.cpp"
#include "../../pwdft_develop_b200/csrc/gemm.hpp"

static std::map<void*, size_t> g_live;
static size_t g_used = 0, g_limit = 0;
static int g_calls = 0;

extern "C" {
cudaError_t CUDARTAPI cudaMalloc(void** p, size_t n) {
  ++g_calls;
  if (g_used + n > g_limit) return cudaErrorMemoryAllocation;
  *p = malloc(1);
  g_live[*p] = n;
  g_used += n;
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaFree(void* p) {
  if (!p) return cudaSuccess;
  g_used -= g_live.at(p);
  g_live.erase(p);
  free(p);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaGetLastError(void) { return cudaSuccess; }
const char* CUDARTAPI cudaGetErrorString(cudaError_t) { return "out of memory"; }
cudaError_t CUDARTAPI cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
}
namespace pwb {
void set_error(const std::string&) {}
}

#define CHECK(x)                                                  \
  do {                                                            \
    if (!(x)) {                                                   \
      std::fprintf(stderr, "line %d: %s\n", __LINE__, #x);        \
      return 1;                                                   \
    }                                                             \
  } while (0)

int main() {
  std::vector<void*> kept;
  {
    pwb::DevBuf b;
    b.keep = &kept;
    g_limit = 100;
    CHECK(b.alloc(40) == PW_OK && b.bytes == 40 && kept.empty());
    void* p = b.p;
    // no room for 70 beside the 40 in use: the 40 stay, nothing is retired
    CHECK(b.alloc(70) == PW_ENOMEM);
    CHECK(b.p == p && b.bytes == 40 && kept.empty() && g_used == 40);
    CHECK(b.alloc(40) == PW_OK && b.p == p);
    // a growth by half does not fit, the request itself does
    g_limit = 95;
    CHECK(b.grow(50) == PW_OK && b.bytes == 50);
    CHECK(kept.size() == 1 && kept[0] == p);
    CHECK(b.grow(60) == PW_ENOMEM && b.bytes == 50 && kept.size() == 1);
    // smaller requests change nothing
    const int calls = g_calls;
    CHECK(b.alloc(10) == PW_OK && b.grow(50) == PW_OK && g_calls == calls && b.bytes == 50);
  }
  for (void* p : kept) cudaFree(p);
  kept.clear();
  CHECK(g_used == 0 && g_live.empty());
  {
    // many small steps: all blocks together stay below three times the last
    pwb::DevBuf b;
    b.keep = &kept;
    g_limit = (size_t)1 << 40;
    for (size_t n = 1000; n < 1000000; n += 1000) CHECK(b.grow(n) == PW_OK && b.bytes >= n);
    CHECK(g_used <= 3 * b.bytes);
    CHECK(b.bytes < 1500000);
  }
  for (void* p : kept) cudaFree(p);
  kept.clear();
  {
    // a block that a capture may have recorded is neither freed by a growth nor given back
    pwb::DevBuf b;
    g_limit = 1000;
    CHECK(b.alloc(60) == PW_OK);
    void* p = b.p;
    b.keep = &kept;
    CHECK(b.alloc(90) == PW_OK && kept.size() == 1 && kept[0] == p && g_live.count(p));
    void* q = b.p;
    b.drop();
    CHECK(!b.p && !b.bytes && kept.size() == 2 && g_live.count(q) && g_used == 150);
    CHECK(b.alloc(30) == PW_OK && b.bytes == 30);
  }
  for (void* p : kept) cudaFree(p);
  {
    // without `keep` the old block is freed before the new one is asked for
    pwb::DevBuf b;
    g_limit = 100;
    CHECK(b.alloc(60) == PW_OK && b.alloc(90) == PW_OK && g_used == 90);
  }
  CHECK(g_used == 0);
  {
    // a batched reduction needs a place for every product
    double x;
    pwb::ReduceOut o;
    o.out = &x;
    CHECK(pwb::reduce_ok(o, 1) && !pwb::reduce_ok(o, 2));
    o.out = nullptr;
    o.bf_hi = &x;
    CHECK(pwb::reduce_ok(o, 1) && !pwb::reduce_ok(o, 2));
    o.bs_bf = 8;
    CHECK(pwb::reduce_ok(o, 65535) && !pwb::reduce_ok(o, 65536) && !pwb::reduce_ok(o, 0));
  }
  std::puts("ok");
  return 0;
}
