// Host check of the growing work buffers with a memory that fails on demand: after a failed growth a buffer holds no
// block that was given back, a smaller request allocates, and a failed call's kept buffers are released.
#include <cstdio>
#include <new>
#include <set>

#include "../cheese_b200/csrc/cz_buf.h"

struct Fake {
  static std::set<void *> live;
  static int fail_in;              // the allocations until one fails; negative: never
  static int bad;
  static void *get(size_t n) {
    if (fail_in == 0) { fail_in = -1; throw std::bad_alloc(); }
    if (fail_in > 0) fail_in--;
    void *p = ::operator new(n);
    live.insert(p);
    return p;
  }
  static void put(void *p) {
    if (!live.erase(p)) { bad++; return; }
    ::operator delete(p);
  }
  static void drop(void *p) { put(p); }
};
std::set<void *> Fake::live;
int Fake::fail_in = -1, Fake::bad = 0;

using Buf = cz::GrowBuf<Fake>;
struct Tree {
  Buf a, b;
  void release() { a.release(); b.release(); }
};

int errors = 0;
void expect(bool ok, const char *what) {
  if (!ok) { errors++; std::printf("%s\n", what); }
}

bool call(Tree &t, size_t n) {     // a call that keeps its buffers for the next one
  try {
    cz::ReleaseUnlessDone<Tree> guard{t};
    t.a.ensure(n);
    t.b.ensure(n);
    guard.done = true;
    return true;
  } catch (const std::bad_alloc &) {
    return false;
  }
}

int main() {
  Buf b;
  b.ensure(1000);
  expect(b.p && b.cap >= 1000 && Fake::live.count(b.p), "first block");
  void *first = b.p;
  b.ensure(900);
  expect(b.p == first, "a smaller request keeps the block");
  Fake::fail_in = 0;
  bool threw = false;
  try { b.ensure(100000); } catch (const std::bad_alloc &) { threw = true; }
  expect(threw && b.p == nullptr && b.cap == 0 && Fake::live.empty(), "a failed growth leaves the buffer empty");
  b.ensure(500);
  expect(b.p && b.cap >= 500 && Fake::live.count(b.p), "a smaller request allocates after the failure");
  b.release();
  b.release();
  expect(Fake::live.empty(), "released");

  Tree t;
  expect(call(t, 2000) && Fake::live.size() == 2, "a call keeps its buffers");
  Fake::fail_in = 1;               // the second buffer's growth fails
  expect(!call(t, 50000) && Fake::live.empty() && !t.a.p && !t.b.p, "a failed call keeps nothing");
  expect(call(t, 100) && Fake::live.size() == 2 && Fake::live.count(t.a.p) && Fake::live.count(t.b.p), "the next call");
  t.release();
  expect(Fake::live.empty() && Fake::bad == 0, "every block given back once");
  std::printf("errors: %d\n", errors);
  return errors != 0;
}
