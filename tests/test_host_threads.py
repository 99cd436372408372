"""The host passes that op_decl_map, op_decl_dat and op_plan_core cut into parts
(csrc/host_threads.h), in a process that cannot have all the threads, or any:
every part runs once all the same and nothing is thrown."""
import os
import subprocess

import pytest

from conftest import ROOT, scratch_dir

SRC = r"""
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>
#include <atomic>
#include "host_threads.h"
static int left;
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x) {
  if (left-- <= 0) return EAGAIN;
  typedef int (*Real)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
  static Real real = (Real)dlsym(RTLD_NEXT, "pthread_create");
  return real(t, a, f, x);
}
int main(int, char **v) {
  left = atoi(v[1]);
  const size_t n = (size_t)atoi(v[2]);
  std::vector<std::atomic<int>> ran(n);
  op2b::on_threads(n, [&](size_t t) { ran[t]++; });
  for (auto &r : ran) printf("%d ", r.load());
  return 0;
}
"""


@pytest.fixture(scope="module")
def exe():
    d = scratch_dir()
    cpp, out = os.path.join(d, "threads.cpp"), os.path.join(d, "threads")
    with open(cpp, "w") as f:
        f.write(SRC)
    csrc = os.path.join(ROOT, "oplus2_matlab_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-I", csrc, cpp, "-o", out, "-pthread", "-ldl"], check=True)
    yield out
    os.remove(cpp)
    os.remove(out)


@pytest.mark.parametrize("parts", [1, 2, 8])
@pytest.mark.parametrize("threads", [0, 1, 3, 100])
def test_every_part_runs_once(exe, threads, parts):
    r = subprocess.run([exe, str(threads), str(parts)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == ["1"] * parts
