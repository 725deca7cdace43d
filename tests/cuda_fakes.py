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
typedef int (*free_t)(void*);
typedef int (*info_t)(size_t*, size_t*);
typedef int (*launch_t)(void*, void*);
typedef int (*elapsed_t)(float*, void*, void*);
#define REAL(type, name) static type real; if (!real) real = (type)dlsym(RTLD_NEXT, name)
static int mallocs = -1, launches = -1;      /* calls that still pass; -1: all */
static size_t at_least = 0;                  /* allocations of at least so many bytes count */
static long long room = -1;                  /* free device memory of a small device; -1: the real one */
static int slow = 0;                         /* event times that come out a thousand times longer */
static struct { void* p; size_t n; } blocks[1 << 16];
static int n_blocks = 0;
void fake_fail_malloc(int after, size_t bytes) { mallocs = after; at_least = bytes; }
void fake_fail_graph_launch(int after) { launches = after; }
void fake_room(long long bytes) { room = bytes; }
long long fake_room_left(void) { return room; }
void fake_slow_events(int n) { slow = n; }
int cudaMalloc(void** p, size_t n) {
    int e;
    REAL(malloc_t, "cudaMalloc");
    if (mallocs >= 0 && n >= at_least && mallocs-- == 0) { mallocs = 0; return 2; }   /* cudaErrorMemoryAllocation */
    if (room >= 0 && (long long)n > room) return 2;
    e = real(p, n);
    if (e == 0 && n_blocks < 1 << 16) { blocks[n_blocks].p = *p; blocks[n_blocks++].n = n; }
    if (e == 0 && room >= 0) room -= (long long)n;
    return e;
}
int cudaFree(void* p) {
    int i;
    REAL(free_t, "cudaFree");
    for (i = 0; p && i < n_blocks; ++i)
        if (blocks[i].p == p) {
            if (room >= 0) room += (long long)blocks[i].n;
            blocks[i] = blocks[--n_blocks];
            break;
        }
    return real(p);
}
int cudaMemGetInfo(size_t* left, size_t* all) {
    int e;
    REAL(info_t, "cudaMemGetInfo");
    e = real(left, all);
    if (e == 0 && room >= 0) *left = (size_t)room;
    return e;
}
int cudaGraphLaunch(void* g, void* s) {
    REAL(launch_t, "cudaGraphLaunch");
    if (launches >= 0 && launches-- == 0) { launches = 0; return 999; }               /* cudaErrorUnknown */
    return real(g, s);
}
int cudaEventElapsedTime(float* ms, void* a, void* b) {
    int e;
    REAL(elapsed_t, "cudaEventElapsedTime");
    e = real(ms, a, b);
    if (slow > 0) { --slow; *ms *= 1000.0f; }
    return e;
}
"""


def run_with_fakes(tmp_path, body):
    """Runs the Python text `body` in a process of its own, with `fakes` (the library above: each
    fake_fail_* call lets that many calls pass and fails the ones after, -1 ends it; fake_room
    leaves that many bytes of device memory free; fake_slow_events lengthens that many event
    times) and the tests' modules at hand."""
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
        fakes.fake_room.argtypes = [ctypes.c_longlong]
        fakes.fake_room_left.restype = ctypes.c_longlong
        """) % ([os.path.join(ROOT, d) for d in ("gdtk-rmhd_b200", "oracle", "tests")], str(so))
    r = subprocess.run([sys.executable, "-c", head + textwrap.dedent(body)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=f"{so} {cudart}"), cwd=ROOT)
    assert r.returncode == 0, r.stdout + r.stderr
