"""Host allocations that fail: each of a plan's creation and of an expansion
formed on request gives the status for memory, not an exception past the C
entry, and the library goes on.  A preloaded operator new fails the k-th
allocation of 256 bytes or more, for every k, in a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

NEW = r"""
#include <atomic>
#include <cstdlib>
#include <new>
static std::atomic<long> left{-1};
extern "C" void oom_arm(long n) { left = n; }
extern "C" long oom_left() { return left; }
static void* get(size_t n) {
  if (n >= 256 && left.load() >= 0 && left.fetch_sub(1) == 0) throw std::bad_alloc();
  if (void* p = malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void* operator new(size_t n) { return get(n); }
void* operator new[](size_t n) { return get(n); }
void operator delete(void* p) noexcept { free(p); }
void operator delete[](void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }
void operator delete[](void* p, size_t) noexcept { free(p); }
"""

RUN = r"""
import ctypes, sys
import numpy as np
import fgt2d_b200 as F
o = ctypes.CDLL(sys.argv[1])
o.oom_arm.argtypes = [ctypes.c_long]
o.oom_left.restype = ctypes.c_long
dim, n = int(sys.argv[2]), int(sys.argv[3])
rng = np.random.default_rng(n)
src, q = rng.random((n, dim)), rng.random((n, 1))
ctx = F.Context(0, host_threads=1)
make = lambda: F.Plan(ctx, dim, 1, 1e-2, 1e-6, src, None, 1, 0)

def sweep(call):
    # call() with the k-th allocation failing, k from 0 on until none is left to fail
    for k in range(5000):
        o.oom_arm(k)
        try:
            got = call()
        except F.FGTError as e:
            assert o.oom_left() < 0 and e.status == 3, e
            continue
        finally:
            failed = o.oom_left() < 0
            o.oom_arm(-1)
        if not failed:
            return k, got
        if hasattr(got, "close"):  # the library did without that allocation
            got.close()
    raise AssertionError("no end")

plan = make()
ref = plan.execute_host(src, q)[0]
T = F.HostTree(dim, 1e-2, 1e-6, src, src[:0])
box = int(np.flatnonzero((T["ilevel"] > max(T["npwlevel"], 0)) & (T["isrcse"].reshape(-1, 2)[:, 1] >= T["isrcse"].reshape(-1, 2)[:, 0]))[0])
mp = plan.expansion("mp", box)
a, again = sweep(lambda: plan.expansion("mp", box))
assert np.array_equal(mp, again)
plan.close()
b, p2 = sweep(make)
assert np.array_equal(p2.execute_host(src, q)[0], ref)
p2.close()
print("allocations:", a, b)
assert a > 0 and b > 20
"""


@pytest.mark.parametrize("dim,n", [(2, 2500), (3, 2900), (2, 6000), (3, 8000)])
def test_failed_allocations(fgt, tmp_path, dim, n):
    (tmp_path / "new.cpp").write_text(NEW)
    so = str(tmp_path / "new.so")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", so, str(tmp_path / "new.cpp")], check=True)
    r = subprocess.run([sys.executable, "-c", RUN, so, str(dim), str(n)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300, env=dict(os.environ, LD_PRELOAD=so))
    print(r.stdout)
    assert r.returncode == 0, r.stderr[-2000:]
