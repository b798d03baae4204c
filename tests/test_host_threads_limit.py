"""The host-thread split (`parallel_indices` in distembed_gb300/csrc/de_internal.h) where
the system gives no or few more threads: the calling thread takes what is left, every index
is visited exactly once, and nothing is thrown at the C entry points that use it.  A
`pthread_create` of the program's own stands in for the limit."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = next((d for d in (os.environ.get("CUDA_HOME", "") + "/include", "/usr/local/cuda/include")
                 if os.path.exists(os.path.join(d, "cuda_runtime.h"))), None)

PROGRAM = r"""
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include "de_internal.h"

static int allowed = 0;
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
  typedef int (*Fn)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
  static Fn real = reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"));
  if (allowed-- <= 0) return EAGAIN;
  return real(t, a, f, arg);
}

int main(int, char **argv) {
  allowed = std::atoi(argv[1]);
  const long long count = 300007;
  std::vector<std::atomic<int>> hits(count);
  for (auto &h : hits) h = 0;
  de::parallel_indices(count, 4, [&](int64_t i) { hits[i].fetch_add(1); });
  for (long long i = 0; i < count; ++i)
    if (hits[i] != 1) { std::printf("index %lld hit %d times\n", i, int(hits[i])); return 1; }
  std::printf("ok\n");
  return 0;
}
"""


@pytest.mark.skipif(CUDA_INC is None or shutil.which("g++") is None, reason="needs g++ and the CUDA headers")
def test_parallel_indices_without_threads_to_be_had(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-D_GNU_SOURCE", "-pthread",
                           "-I", os.path.join(ROOT, "distembed_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
                           "-I", CUDA_INC, str(src), "-o", str(exe), "-ldl"])
    for allowed in (0, 1, 3, 1000):
        r = subprocess.run([str(exe), str(allowed)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0 and r.stdout.strip() == "ok", (allowed, r.stdout + r.stderr)
