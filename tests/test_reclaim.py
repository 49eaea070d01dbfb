"""dv_reclaim.h: what holders keep goes back when it is asked for, for one device,
from any thread, also where one holder owns another, and a holder that is gone
is not asked."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <stdio.h>
#include <atomic>
#include <memory>
#include <thread>
#include "dv_reclaim.h"
using namespace dv;
struct Spare final : Holder {  // as an engine's freed blocks
  size_t bytes;
  int device;
  Spare(size_t b, int d) : bytes(b), device(d) { Holders::add(this); }
  ~Spare() { Holders::remove(this); }
  size_t reclaim(int d) override {
    const size_t b = d == device ? bytes : 0;
    if (d == device) bytes = 0;
    return b;
  }
};
struct Parked final : Holder {  // as an idle server's engine, with freed blocks of its own
  std::unique_ptr<Spare> e;
  Parked() { Holders::add(this); }
  ~Parked() { Holders::remove(this); }
  void put(std::unique_ptr<Spare> x) {
    std::lock_guard<std::recursive_mutex> g(Holders::lock());
    e = std::move(x);
  }
  std::unique_ptr<Spare> take() {
    std::lock_guard<std::recursive_mutex> g(Holders::lock());
    return std::move(e);
  }
  size_t reclaim(int d) override {
    if (!e || e->device != d) return 0;
    const size_t b = e->bytes;
    e.reset();
    return b;
  }
};
int main() {
  if (Holders::reclaim_all(0) != 0) return 1;
  Spare a(100, 0), b(30, 1);
  {
    Spare gone(7, 0);
  }
  if (Holders::reclaim_all(0) != 100 || a.bytes != 0 || b.bytes != 30) return 2;
  Parked p;  // registered before and after what it owns
  p.put(std::make_unique<Spare>(50, 0));
  if (Holders::reclaim_all(1) != 30 || !p.e) return 3;
  if (Holders::reclaim_all(0) != 50 || p.take()) return 4;
  auto early = std::make_unique<Spare>(60, 0);
  Parked q;
  q.put(std::move(early));
  if (Holders::reclaim_all(0) != 60 || q.take()) return 5;
  // one thread parks and takes, another asks: nothing is lost or given twice
  std::atomic<bool> stop{false};
  size_t given = 0, kept = 0, made = 0;
  std::thread t([&] { while (!stop) given += Holders::reclaim_all(0); });
  for (int i = 0; i < 20000; ++i) {
    p.put(std::make_unique<Spare>(1, 0));
    ++made;
    if (auto e = p.take()) {
      std::lock_guard<std::recursive_mutex> g(Holders::lock());
      kept += e->bytes;
      e->bytes = 0;
    }
  }
  stop = true;
  t.join();
  return given + kept == made ? 0 : 6;
}
"""


def test_holders_give_back(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-pthread", "-fsanitize=address,undefined", "-I",
                           os.path.join(ROOT, "dvide_b200", "csrc"), str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, (out.returncode, out.stderr[-2000:])
