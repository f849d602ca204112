// The split engine's buffers (ballasim_b200/csrc/split_bufs.h) over a fake device memory that refuses allocations:
// exits 0 where the named check holds, else prints what does not.
#include <cstdio>
#include <cstring>
#include <set>

#include "split_bufs.h"

namespace {

struct Refused {};

// Every allocation live now; an allocation of more than `most` is refused.
std::set<const void*> live;
size_t most = 0;
int failures = 0;

struct FakeBuf {
  char* p = nullptr;
  size_t cap = 0;
  void release() {
    live.erase(p);
    delete[] p;
    p = nullptr;
    cap = 0;
  }
  ~FakeBuf() { release(); }
  void ensure(size_t n) {
    if (n <= cap && p) return;
    release();
    if (n > most) throw Refused{};
    p = new char[n];
    cap = n;
    live.insert(p);
  }
};
using Bufs = bs::SplitBufs<FakeBuf, FakeBuf, FakeBuf>;

#define CHECK(x)                                             \
  do {                                                       \
    if (!(x)) {                                              \
      std::printf("%s:%d: %s\n", __FILE__, __LINE__, #x);    \
      ++failures;                                            \
    }                                                        \
  } while (0)

template <class F>
bool refused(F&& f) {
  try {
    f();
  } catch (const Refused&) {
    return true;
  }
  return false;
}

// A list that could not grow has no capacity: the smaller shape afterwards allocates again.
void refused_list() {
  Bufs b;
  most = 1000;
  b.ensure(10, 8, 100, 2);
  CHECK(b.capacity == 8 && live.count(b.rest.p) == 1);
  CHECK(refused([&] { b.ensure(10, 11, 100, 2); }));
  CHECK(b.capacity == 0 && b.rest.p == nullptr);
  b.ensure(10, 8, 100, 2);
  CHECK(b.capacity == 8 && b.rest.cap >= 800 && live.count(b.rest.p) == 1);
  b.release();
  CHECK(b.capacity == 0 && live.empty());
  b.ensure(10, 3, 100, 2);
  CHECK(b.capacity == 3 && b.rest.cap >= 300 && live.count(b.rest.p) == 1);
}

}  // namespace

int main(int argc, char** argv) {
  const char* name = argc > 1 ? argv[1] : "";
  if (!std::strcmp(name, "refused_list")) refused_list();
  else return 2;
  return failures ? 1 : 0;
}
