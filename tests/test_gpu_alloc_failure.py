"""Device allocations that fail: a stand-in for cudaMalloc that refuses large
requests, preloaded into a child process (no device memory is filled)."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
FAKE = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static size_t from = (size_t)-1;
static int refusals = 0;
void fake_refuse_from(size_t n) { from = n; }
int fake_refusals(void) { return refusals; }
int cudaMalloc(void** p, size_t n) {
   static int (*real)(void**, size_t) = 0;
   if (!real) {
      void* lib = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
      real = lib ? (int (*)(void**, size_t))dlsym(lib, "cudaMalloc") : 0;
      if (!real) return 999;
   }
   if (n >= from) {
      ++refusals;
      return real(p, (size_t)1 << 60);
   }
   return real(p, n);
}
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d = tmp_path_factory.mktemp("fake")
    src, so = d / "fake.c", d / "libfakemalloc.so"
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(so), "-ldl"], check=True)
    return str(so)


@pytest.mark.parametrize("what", ["reserve", "create", "sweep"])
def test_refused_allocation(fake, what):
    env = dict(os.environ, LD_PRELOAD=fake)
    res = subprocess.run([sys.executable, os.path.join(HERE, "alloc_failure_child.py"), what, fake],
                         capture_output=True, text=True, timeout=300, env=env)
    assert res.returncode == 0 and res.stdout.strip().endswith("ok"), res.stdout + res.stderr
