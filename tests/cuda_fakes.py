"""Failing CUDA runtime calls for the tests of error paths: a library loaded before libcudart
answers the calls it is told to with an error code and passes all others on, so that the
library under test sees a failed allocation or launch and the GPU sees nothing."""
import os
import subprocess
import sys
import textwrap

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
typedef int (*malloc_t)(void**, size_t);
typedef int (*launch_t)(void*, void*);
static int mallocs = -1, launches = -1;      /* calls that still pass; -1: all */
static size_t at_least = 0;                  /* allocations of at least so many bytes count */
void fake_fail_malloc(int after, size_t bytes) { mallocs = after; at_least = bytes; }
void fake_fail_graph_launch(int after) { launches = after; }
int cudaMalloc(void** p, size_t n) {
    static malloc_t real;
    if (!real) real = (malloc_t)dlsym(RTLD_NEXT, "cudaMalloc");
    if (mallocs >= 0 && n >= at_least && mallocs-- == 0) { mallocs = 0; return 2; }   /* cudaErrorMemoryAllocation */
    return real(p, n);
}
int cudaGraphLaunch(void* g, void* s) {
    static launch_t real;
    if (!real) real = (launch_t)dlsym(RTLD_NEXT, "cudaGraphLaunch");
    if (launches >= 0 && launches-- == 0) { launches = 0; return 999; }               /* cudaErrorUnknown */
    return real(g, s);
}
"""


def run_with_fakes(tmp_path, body):
    """Runs the Python text `body` in a process of its own, with `fakes` (the library above: each
    fake_fail_* call lets that many calls pass and fails the ones after, -1 ends it) and the
    tests' modules at hand."""
    src, so = tmp_path / "fakes.c", tmp_path / "fakes.so"
    src.write_text(SOURCE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(so), str(src), "-ldl"], check=True)
    find = ("import torch, re; torch.cuda.is_available(); "
            "print(sorted(set(re.findall(r'/\\S*libcudart\\S*', open('/proc/self/maps').read())))[0])")
    cudart = subprocess.run([sys.executable, "-c", find], check=True, capture_output=True, text=True).stdout.strip()
    head = textwrap.dedent("""
        import ctypes, sys
        sys.path[:0] = %r
        fakes = ctypes.CDLL(%r)
        fakes.fake_fail_malloc.argtypes = [ctypes.c_int, ctypes.c_size_t]
        """) % ([os.path.join(ROOT, d) for d in ("gdtk-rmhd_b200", "oracle", "tests")], str(so))
    r = subprocess.run([sys.executable, "-c", head + textwrap.dedent(body)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=f"{so} {cudart}"), cwd=ROOT)
    assert r.returncode == 0, r.stdout + r.stderr
