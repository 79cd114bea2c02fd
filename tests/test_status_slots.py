"""The pool of page-locked status slots (csrc/slot_pool.hpp): on the CPU against an allocator whose memory goes
with its context, as the runtime's does on a device reset, and on the GPU with such a reset between two handles."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "multifrontal-dag_b200", "csrc")

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <thread>
#include "slot_pool.hpp"
struct Fake {                                  // contexts of two devices, memory that dies with its context
  struct Mem { size_t bytes; unsigned long long ctx; };
  static unsigned long long id[2], last;
  static thread_local int cur;
  static std::map<char*, Mem> live;
  static bool fails;
  static unsigned long long context() { return id[cur]; }
  static void* lock(size_t n) {
    if (fails) return nullptr;
    char* p = (char*)std::malloc(n);
    live[p] = {n, id[cur]};
    return p;
  }
  static void unlock(void* p) {
    if (!live.erase((char*)p)) { std::puts("unlock of memory that is not there"); std::exit(1); }
  }
  static void reset(int d) {
    for (auto it = live.begin(); it != live.end();) it = it->second.ctx == id[d] ? live.erase(it) : std::next(it);
    id[d] = ++last;
  }
  static bool alive(void* q, size_t n) {
    for (auto& m : live) if ((char*)q >= m.first && (char*)q + n <= m.first + m.second.bytes) return true;
    return false;
  }
};
unsigned long long Fake::id[2] = {1, 2}, Fake::last = 2;
thread_local int Fake::cur = 0;
std::map<char*, Fake::Mem> Fake::live;
bool Fake::fails = false;
using Pool = mfd::SlotPool<Fake>;
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int reset() {                                  // a slot taken after a reset is in memory of the new context
  Pool p;
  Fake::cur = 0;
  Pool::Slot a = p.take(0), b = p.take(0);
  CHECK(Fake::alive(a.p, 256) && Fake::alive(b.p, 256));
  p.give(a);
  Fake::reset(0);
  Pool::Slot c = p.take(0);
  CHECK(Fake::alive(c.p, 256));
  p.give(b);                                   // of the old context: not handed out again
  for (int k = 0; k < 600; ++k) CHECK(Fake::alive(p.take(0).p, 256));
  return 0;
}
int other_device() {                           // a reset of one device leaves the other's slots alone
  Pool p;
  Fake::cur = 0;
  Pool::Slot a = p.take(0);
  Fake::cur = 1;
  Pool::Slot b = p.take(1);
  Fake::reset(0);
  CHECK(Fake::alive(b.p, 256));
  p.give(b);
  CHECK(Fake::alive(p.take(1).p, 256));
  p.give(a);
  Fake::cur = 0;
  CHECK(Fake::alive(p.take(0).p, 256));
  return 0;
}
int many() {                                   // all distinct; at most one block stays when they are back
  Pool p;
  std::vector<Pool::Slot> s;
  for (int k = 0; k < 1000; ++k) {
    s.push_back(p.take(0));
    CHECK(Fake::alive(s.back().p, 256));
    std::memset(s.back().p, k & 255, 256);
  }
  for (int k = 0; k < 1000; ++k) CHECK(*(unsigned char*)s[k].p == (k & 255));
  for (auto& x : s) p.give(x);
  CHECK(Fake::live.size() <= 1);
  return 0;
}
int no_memory() {                              // refused, and well again afterwards
  Pool p;
  Fake::fails = true;
  Pool::Slot a = p.take(0);
  CHECK(a.p == nullptr);
  p.give(a);
  Fake::fails = false;
  CHECK(Fake::alive(p.take(0).p, 256));
  return 0;
}
int threads() {
  static Pool p;
  static std::atomic<int> bad{0};
  std::vector<std::thread> t;
  for (int k = 0; k < 8; ++k)
    t.emplace_back([k] {
      for (int i = 0; i < 20000; ++i) {
        Pool::Slot s = p.take(0);
        auto* w = static_cast<std::atomic<int>*>(s.p);
        w->store(k);
        if (w->load() != k) ++bad;
        p.give(s);
      }
    });
  for (auto& x : t) x.join();
  CHECK(bad == 0);
  return 0;
}
int main(int, char** argv) {
  const std::string n = argv[1];
  return n == "reset" ? reset() : n == "other_device" ? other_device() : n == "many" ? many() : n == "no_memory" ? no_memory() : threads();
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("slots")
    (d / "main.cpp").write_text("#include <string>\n" + PROGRAM)
    exe = str(d / "main")
    subprocess.run(["g++", "-std=c++17", "-O1", "-D_GLIBCXX_ASSERTIONS", "-pthread", "-I", CSRC, str(d / "main.cpp"), "-o", exe],
                   check=True)
    return exe


@pytest.mark.parametrize("what", ["reset", "other_device", "many", "no_memory", "threads"])
def test_slots(program, what):
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


HANDLES = r"""
import ctypes, sys
from mfdag import hppllt as H, problems as P
p = P.laplace2d(20)
for k in range(3):
    s = H.Solver.analyze(p.n, p.col, p.row, p.order, max_zero=10)
    assert s.factorize(p.val) == 0
    x = p.rhs.copy()
    rep, rc = s.solve(x)
    assert rc == 0 and P.backward_error(p.n, p.col, p.row, p.val, x, p.rhs) <= 1e-12
    s.close()
    rt = ctypes.CDLL("/usr/local/cuda/lib64/libcudart.so.12")
    assert rt.cudaSetDevice(0) == 0 and rt.cudaDeviceReset() == 0
print("handles ok")
"""


@pytest.mark.gpu
def test_new_handle_after_device_reset():
    """A process of its own resets its context between handles: each handle factors and solves."""
    env = dict(os.environ, PYTHONPATH=os.path.join(ROOT, "multifrontal-dag_b200"))
    r = subprocess.run([sys.executable, "-c", HANDLES], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0 and "handles ok" in r.stdout, r.stdout + r.stderr
