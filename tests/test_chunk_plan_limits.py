"""The chunk search where the host gives it no threads or no memory: the same
plan with however many threads start, and MFG_ERR_NOMEM, never an exception or
an abort out of the C entry, where an allocation fails.  pthread_create and
operator new are interposed in a process of its own."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

SHIM = r"""
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <stdlib.h>
#include <atomic>
#include <new>
// threads and allocations still allowed; negative: any number
static std::atomic<long> threads{-1}, news{-1};
static std::atomic<long> refused{0};
static bool take(std::atomic<long> &left) {
  long k = left.load();
  while (k > 0 && !left.compare_exchange_weak(k, k - 1)) {}
  if (k == 0) refused++;
  return k != 0;
}
extern "C" {
void allow(long t, long n) { threads = t; news = n; refused = 0; }
long refusals() { return refused; }
int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x) {
  using fn = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
  static fn real = (fn)dlsym(RTLD_NEXT, "pthread_create");
  return take(threads) ? real(t, a, f, x) : EAGAIN;
}
}
void *operator new(size_t n) {
  void *p = take(news) ? malloc(n ? n : 1) : nullptr;
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }
"""

RUN = r"""
import ctypes, sys
sys.path[:0] = [{here!r}, {root!r}]
from test_chunk_plan import plan, sweep_tables
shim = ctypes.CDLL({shim!r})
shim.allow.argtypes = [ctypes.c_long, ctypes.c_long]
shim.refusals.restype = ctypes.c_long
t = sweep_tables(7)

def planned(force, threads=-1, news=-1):
    shim.allow(threads, news)
    got = plan(t, 60, 16, force)
    n = shim.refusals()
    shim.allow(-1, -1)
    return got, n

def same(a, b):
    return a[0] == b[0] and a[2:] == b[2:] and (a[1] == b[1]).all()

for force in (-1, 0, 1, 4):
    want, _ = planned(force)
    assert want[0] >= 0
    if {what!r} == "threads":
        for k in range(30):
            got, n = planned(force, threads=k)
            assert same(got, want), (force, k)
            if n == 0:
                break
    else:
        k, failed = 0, 0
        while True:
            got, n = planned(force, news=k)
            # (a thread or a sort's buffer that is not had is done without)
            assert same(got, want) or (n > 0 and got[0] == -3), (force, k, got[0])
            failed += got[0] == -3
            if n == 0:
                break
            k += 1 + k // 8
        assert failed > 0
print("done")
"""


@pytest.mark.parametrize("what", ["threads", "memory"])
def test_search_without_threads_or_memory(what, tmp_path):
    src, shim = tmp_path / "shim.cpp", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", str(shim), str(src), "-ldl"],
                   check=True)
    code = RUN.format(here=HERE, root=os.path.dirname(HERE), shim=str(shim), what=what)
    p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=str(shim)))
    assert p.returncode == 0 and p.stdout.strip() == "done", (p.returncode, p.stderr[-2000:])
