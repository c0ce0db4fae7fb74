/* host_copy.h on the host, over fake_cuda/cuda_runtime.h: `host_copy_check
   <check>` prints what failed and returns the number of failures. */
#include "host_copy.h"

#include <cstdio>
#include <ctime>
#include <string>

static int failed = 0;

#define CHECK(x)                                         \
  do {                                                   \
    if (!(x)) {                                          \
      std::printf("line %d: %s\n", __LINE__, #x);        \
      failed++;                                          \
    }                                                    \
  } while (0)

static const size_t MB = (size_t)1 << 20;

/* a read of n bytes gives them */
static void read(size_t n) {
  std::vector<uint8_t> src(n), dst(n);
  for (size_t i = 0; i < n; i += 997) src[i] = (uint8_t)(i / 997);
  src[n - 1] = 77;
  CHECK(host_copy::to_host(dst.data(), src.data(), n, 0) == cudaSuccess);
  CHECK(src == dst);
}

/* a read queued behind half a second of work: no thread works meanwhile */
static void waiting() {
  host_copy::Users u;
  read(40 * MB);
  std::vector<uint8_t> src(40 * MB, 1), dst(40 * MB);
  fake::busy_until = fake::clock::now() + std::chrono::milliseconds(500);
  const std::clock_t c0 = std::clock(); /* of all threads */
  host_copy::to_host(dst.data(), src.data(), src.size(), 0);
  const double cpu = (double)(std::clock() - c0) / CLOCKS_PER_SEC;
  CHECK(fake::clock::now() >= fake::busy_until);
  CHECK(src == dst);
  std::printf("%.3f s of CPU time\n", cpu);
  CHECK(cpu < 0.25);
}

/* the chunks are allocated by a read that gains what they cost, or after as
   many smaller ones as together would have, and go with the last handle */
static void chunks() {
  for (int round = 0; round < 2; ++round) {
    host_copy::Users u;
    const int a0 = fake::allocs, f0 = fake::frees;
    for (int k = 0; k < 24; ++k) read(8 * MB); /* 192 MB */
    read(5 * MB);                              /* not a large read */
    CHECK(fake::allocs == a0);
    read(8 * MB);
    CHECK(fake::allocs == a0 + 2);
    read(8 * MB);
    read(40 * MB);
    CHECK(fake::allocs == a0 + 2);
    CHECK(fake::frees == f0);
  }
  CHECK(fake::locked.empty());
  {
    host_copy::Users u;
    const int a0 = fake::allocs;
    read(31 * MB);
    CHECK(fake::allocs == a0);
    read(32 * MB);
    CHECK(fake::allocs == a0 + 2);
  }
  CHECK(fake::locked.empty());
  host_copy::Users u;
  fake::refuse = true;
  read(40 * MB);
  CHECK(cudaGetLastError() == cudaSuccess);
  fake::refuse = false;
  read(40 * MB);
  CHECK(fake::locked.size() == 2);
}

/* small buffers: of a handle that is gone for the next one, a few of them; not
   what a reset of the device took away; of ordinary memory without any other */
static void small() {
  void* p;
  {
    host_copy::Users u;
    p = host_copy::take_small();
    host_copy::give_small(p);
  }
  CHECK(fake::allocs == 1 && fake::frees == 0);
  {
    host_copy::Users u;
    CHECK(host_copy::take_small() == p);
    host_copy::give_small(p);
    std::vector<void*> many;
    for (int k = 0; k < 20; ++k) many.push_back(host_copy::take_small());
    CHECK(fake::allocs == 20);
    for (void* x : many) host_copy::give_small(x);
  }
  CHECK(fake::locked.size() == 8 && fake::frees == 12);
  fake::locked.clear(); /* cudaDeviceReset, and another buffer where one of them was */
  fake::locked.insert(p);
  std::memset(p, 0, host_copy::kSmall);
  host_copy::Users u;
  p = host_copy::take_small();
  CHECK(fake::allocs == 21 && fake::locked.size() == 2);
  fake::refuse = true;
  void* q = host_copy::take_small();
  CHECK(q != nullptr && q != p && fake::locked.count(q) == 0);
  if (q) std::memset(q, 1, host_copy::kSmall);
  CHECK(cudaGetLastError() == cudaSuccess);
  host_copy::give_small(q);
  host_copy::give_small(p);
  fake::refuse = false;
  CHECK(host_copy::take_small() == p);
  host_copy::give_small(p);
  host_copy::give_small(nullptr);
  static const int gone[4] = {0};
  host_copy::give_small(const_cast<int*>(gone)); /* of a reset while the handle lived: not written to */
  CHECK(cudaGetLastError() == cudaSuccess);
}

int main(int argc, char** argv) {
  const std::string check = argc > 1 ? argv[1] : "";
  if (check == "waiting") waiting();
  else if (check == "chunks") chunks();
  else if (check == "small") small();
  else failed = 100;
  return failed;
}
