// Checks of HostStage (csrc/hostcopy.cuh) against tests/fake_cuda/cuda_runtime.h.
// Prints the first check that does not hold and exits 1.
#include "../../prlgt2020_b200/csrc/hostcopy.cuh"

#include <cstdio>
#include <vector>

using namespace nspt;

#define HOLDS(x)                                         \
  do {                                                   \
    if (!(x)) {                                          \
      printf("line %d does not hold: %s\n", __LINE__, #x); \
      exit(1);                                           \
    }                                                    \
  } while (0)

static std::vector<char> pattern(size_t n, int seed) {
  std::vector<char> v(n);
  for (size_t i = 0; i < n; i++) v[i] = (char)(i * 2654435761u >> 13 ^ seed);
  return v;
}

int main() {
  FakeStream s0 = {0}, s1 = {1};
  {  // whole, both ways, at sizes around the chunks; the caller's device stays
    HostStage h;
    h.user(1);
    size_t asked = 0;
    for (size_t n : {(size_t)1, COPY_LEAST - 1, COPY_LEAST, COPY_LEAST + 1,
                     (size_t)28713984, (size_t)70000001, (size_t)300000007}) {
      const auto a = pattern(n, 1);
      std::vector<char> d(n), b(n);
      Fake::device = 0;
      HOLDS(h.copy(&s1, 1, (void *)a.data(), d.data(), n, false) == cudaSuccess);
      HOLDS(Fake::device == 0);
      HOLDS(h.copy(&s1, 1, b.data(), d.data(), n, true) == cudaSuccess);
      HOLDS(Fake::device == 0);
      HOLDS(d == a && b == a);
      HOLDS(Fake::wrong_device == 0 && Fake::events == 0);
      // one set, once 128 MB have been asked for
      if (n >= COPY_LEAST) asked += 2 * n;
      HOLDS(Fake::pinned.size() == (asked >= COPY_PAYS) && Fake::allocs == (asked >= COPY_PAYS));
    }
    HOLDS(Fake::pinned_bytes == (16u << 20));
    // a smaller copy uses the set that is there
    const int allocs = Fake::allocs;
    const auto a = pattern(COPY_LEAST, 2);
    std::vector<char> d(COPY_LEAST);
    HOLDS(h.copy(&s0, 0, (void *)a.data(), d.data(), a.size(), false) == cudaSuccess);
    HOLDS(d == a && Fake::allocs == allocs);
    h.user(1);
    h.user(-1);
    HOLDS(Fake::pinned.size() == 1);
    h.user(-1);
    HOLDS(Fake::pinned.empty());  // given back with the last user
  }
  {  // a few copies do not pay for a set, more of them do; and anew after a release
    HostStage h;
    const auto a = pattern(COPY_LEAST, 3);
    std::vector<char> d(COPY_LEAST);
    for (int rep = 0; rep < 2; rep++) {
      h.user(1);
      const int allocs = Fake::allocs;
      for (int i = 0; i < 9; i++) {
        HOLDS(h.copy(&s0, 0, (void *)a.data(), d.data(), a.size(), false) == cudaSuccess);
        HOLDS(Fake::allocs == allocs + (i >= 7) && d == a);
      }
      h.user(-1);
    }
  }
  {  // several threads at once, on two devices: one has the set, the others do without
    HostStage h;
    h.user(4);
    const size_t n = 40000003;
    std::vector<std::thread> th;
    std::vector<int> good(4, 0);
    for (int t = 0; t < 4; t++)
      th.emplace_back([&, t] {
        Fake::device = t & 1;
        const auto a = pattern(n, t);
        std::vector<char> d(n), b(n);
        FakeStream *s = t & 2 ? &s1 : &s0;
        for (int rep = 0; rep < 3; rep++) {
          if (h.copy(s, s->device, (void *)a.data(), d.data(), n, false) != cudaSuccess) return;
          if (h.copy(s, s->device, b.data(), d.data(), n, true) != cudaSuccess) return;
          if (d != a || b != a || Fake::device != (t & 1)) return;
        }
        good[t] = 1;
      });
    for (auto &t : th) t.join();
    HOLDS(good == std::vector<int>(4, 1));
    HOLDS(Fake::wrong_device == 0 && Fake::events == 0);
    h.user(-4);
    HOLDS(Fake::pinned.empty());
  }
  {  // an error of any copy comes back, and the next copy is whole
    HostStage h;
    h.user(1);
    const size_t n = 140000003;
    const auto a = pattern(n, 5);
    std::vector<char> d(n);
    for (int at : {0, 5, 66}) {
      Fake::copies = 0;
      Fake::fail_copy = at;
      HOLDS(h.copy(&s0, 0, (void *)a.data(), d.data(), n, false) == cudaErrorInvalidValue);
      Fake::fail_copy = -1;
      HOLDS(h.copy(&s0, 0, (void *)a.data(), d.data(), n, false) == cudaSuccess && d == a);
      HOLDS(Fake::events == 0);
    }
    h.user(-1);
  }
  {  // no pinned memory: the driver's way, in one copy; pinned fields always go that way
    HostStage h;
    h.user(1);
    const size_t n = 140000003;
    const auto a = pattern(n, 6);
    std::vector<char> d(n);
    Fake::fail_alloc = true;
    Fake::copies = 0;
    HOLDS(h.copy(&s1, 1, (void *)a.data(), d.data(), n, false) == cudaSuccess && d == a);
    HOLDS(Fake::copies == 1);
    Fake::fail_alloc = false;
    void *p;
    cudaHostAlloc(&p, n, 0);
    memcpy(p, a.data(), n);
    Fake::copies = 0;
    HOLDS(h.copy(&s1, 1, p, d.data(), n, false) == cudaSuccess && d == a);
    HOLDS(Fake::copies == 1 && Fake::wrong_device == 0);
    cudaFreeHost(p);
    h.user(-1);
  }
  printf("ok\n");
  return 0;
}
