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
  const auto none = [] {};
  most = 1000;
  b.ensure(10, 8, 100, 2, none);
  CHECK(b.capacity == 8 && live.count(b.rest.p) == 1);
  CHECK(refused([&] { b.ensure(10, 11, 100, 2, none); }));
  CHECK(b.capacity == 0 && b.rest.p == nullptr);
  b.ensure(10, 8, 100, 2, none);
  CHECK(b.capacity == 8 && b.rest.cap >= 800 && live.count(b.rest.p) == 1);
  b.release();
  CHECK(b.capacity == 0 && live.empty());
  b.ensure(10, 3, 100, 2, none);
  CHECK(b.capacity == 3 && b.rest.cap >= 300 && live.count(b.rest.p) == 1);
}

// What a captured step holds is live as long as the step is: it goes before any buffer of its moves, a refused one too.
void captured_addresses() {
  Bufs b;
  const void* held[3] = {nullptr, nullptr, nullptr};
  bool captured = false;
  const auto holds_live = [&] {
    for (const void* q : held) CHECK(live.count(q) == 1);
  };
  const auto drop = [&] {
    if (captured) holds_live();
    captured = false;
  };
  const auto step = [&](size_t scratch, unsigned slots, size_t windows, bool graph) {
    b.ensure(scratch, slots, 100, windows, drop);
    if (graph && !captured) {
      held[0] = b.scratch.p;
      held[1] = b.rest.p;
      held[2] = b.counts.p;
      captured = true;
    }
    if (captured) holds_live();
  };
  most = 1000;
  for (const size_t scratch : {size_t{10}, size_t{40}}) {
    for (const unsigned slots : {4u, 9u}) {
      for (const size_t windows : {size_t{10}, size_t{60}}) {
        step(10, 4, 10, true);
        step(scratch, slots, windows, false);
        step(10, 4, 10, true);
        CHECK(refused([&] { step(10, 11, 10, false); }));
        CHECK(!captured);
        step(10, 4, 10, true);
        CHECK(captured);
        drop();
        b.release();
      }
    }
  }
  b.ensure(10, 4, 100, 10, drop);
  int moves = 0;
  b.ensure(9, 3, 100, 10, [&] { ++moves; });
  CHECK(moves == 0);  // nothing moves for a call that fits
}

// A need that does not fit beside the buffers: they give way once, and what is refused after that is refused.
void gives_way() {
  Bufs b;
  most = 1000;
  b.ensure(10, 8, 100, 2, [] {});
  CHECK(!b.empty());
  FakeBuf events;
  int tries = 0, given = 0;
  const auto need = [&](size_t n) {
    return [&, n] {
      ++tries;
      most = b.empty() ? 2000 : 1000;
      events.ensure(n);
    };
  };
  const auto give = [&] {
    if (b.empty()) return false;
    b.release();
    ++given;
    return true;
  };
  bs::with_room<Refused>(need(900), give);
  CHECK(tries == 1 && given == 0 && events.cap == 900);
  bs::with_room<Refused>(need(1500), give);
  CHECK(tries == 3 && given == 1 && events.cap == 1500 && b.empty());
  CHECK(refused([&] { bs::with_room<Refused>(need(3000), give); }));
  CHECK(tries == 4 && given == 1 && events.p == nullptr);
}

}  // namespace

int main(int argc, char** argv) {
  const char* name = argc > 1 ? argv[1] : "";
  if (!std::strcmp(name, "refused_list")) refused_list();
  else if (!std::strcmp(name, "captured_addresses")) captured_addresses();
  else if (!std::strcmp(name, "gives_way")) gives_way();
  else return 2;
  return failures ? 1 : 0;
}
