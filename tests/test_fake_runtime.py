"""Host paths that only a failing CUDA call reaches, on a fake CUDA runtime: a
small C library with the runtime's entry points, loaded before libcudart, in a
process of its own.  Its device memory is host memory that nothing touches, its
launches do nothing, and it fails the calls that a test names."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#include <stdio.h>
#include <stdlib.h>
typedef int err_t;
typedef struct { unsigned x, y, z; } dim3_t;
static int last = 0, fail_launch = 0;
static size_t fail_size = 0, biggest_ok = 0;
static size_t sizes[4096];
static int n_sizes = 0;
/* controls */
void fake_fail_launches(int n) { fail_launch = n; }
void fake_fail_malloc(size_t bytes) { fail_size = bytes; }
int fake_mallocs_of(size_t bytes) { int k = 0; for (int i = 0; i < n_sizes; ++i) k += sizes[i] == bytes; return k; }
int fake_last_error(void) { return last; }
/* the runtime */
err_t cudaMalloc(void** p, size_t n) {
  if (n == fail_size) { *p = 0; return last = 2; }
  if (n_sizes < 4096) sizes[n_sizes++] = n;
  *p = malloc(64);
  return 0;
}
err_t cudaFree(void* p) { free(p); return 0; }
err_t cudaHostAlloc(void** p, size_t n, unsigned f) { (void)f; *p = calloc(1, n); return 0; }
err_t cudaMallocHost(void** p, size_t n) { *p = calloc(1, n); return 0; }
err_t cudaFreeHost(void* p) { free(p); return 0; }
err_t cudaMemcpyAsync(void* d, const void* s, size_t n, int k, void* st) { (void)d; (void)s; (void)n; (void)k; (void)st; return 0; }
err_t cudaMemsetAsync(void* d, int v, size_t n, void* st) { (void)d; (void)v; (void)n; (void)st; return 0; }
err_t cudaStreamCreateWithFlags(void** s, unsigned f) { (void)f; *s = malloc(8); return 0; }
err_t cudaStreamDestroy(void* s) { free(s); return 0; }
err_t cudaStreamSynchronize(void* s) { (void)s; return 0; }
err_t cudaStreamWaitEvent(void* s, void* e, unsigned f) { (void)s; (void)e; (void)f; return 0; }
err_t cudaEventCreate(void** e) { *e = malloc(8); return 0; }
err_t cudaEventCreateWithFlags(void** e, unsigned f) { (void)f; *e = malloc(8); return 0; }
err_t cudaEventDestroy(void* e) { free(e); return 0; }
err_t cudaEventRecord(void* e, void* s) { (void)e; (void)s; return 0; }
err_t cudaEventSynchronize(void* e) { (void)e; return 0; }
err_t cudaGetDevice(int* d) { *d = 0; return 0; }
err_t cudaDeviceGetAttribute(int* v, int a, int d) { (void)a; (void)d; *v = 152; return 0; }
err_t cudaFuncSetAttribute(const void* f, int a, int v) { (void)f; (void)a; (void)v; return 0; }
err_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int b, size_t s) { (void)f; (void)b; (void)s; *n = 4; return 0; }
err_t cudaGetLastError(void) { int e = last; last = 0; return e; }
static err_t launch(void) {
  if (fail_launch > 0) { --fail_launch; return last = 9; }
  return 0;
}
err_t cudaLaunchKernelExC(const void* c, const void* f, void** a) { (void)c; (void)f; (void)a; return launch(); }
err_t __cudaLaunchKernel(void* f, dim3_t g, dim3_t b, void** a, size_t s, void* st) { (void)f; (void)g; (void)b; (void)a; (void)s; (void)st; return launch(); }
err_t cudaLaunchKernel(const void* f, dim3_t g, dim3_t b, void** a, size_t s, void* st) { (void)f; (void)g; (void)b; (void)a; (void)s; (void)st; return launch(); }
err_t __cudaGetKernel(void** k, const void* f) { *k = (void*)f; return 0; }
"""

PRELUDE = r"""
import ctypes, sys
sys.path.insert(0, {root!r})
fake = ctypes.CDLL({fake!r})
fake.fake_mallocs_of.argtypes = [ctypes.c_size_t]
fake.fake_fail_malloc.argtypes = [ctypes.c_size_t]
import importlib.util, types
pkg = types.ModuleType("gpt_gb300"); pkg.__path__ = [{root!r} + "/gpt_gb300"]
sys.modules["gpt_gb300"] = pkg  # the binding alone: torch would load its own runtime
from gpt_gb300 import _lib
L = _lib.load()
P = ctypes.c_void_p

def create(name, prec, dims, Ls=1, n_rhs=1):
    p = _lib.gbf_params()
    for i, d in enumerate(dims):
        p.dims[i] = d
    p.Ls, p.n_rhs, p.mass, p.xi_0, p.nu, p.reconstruct = Ls, n_rhs, 0.1, 1.0, 1.0, -1
    p.mass_plus = p.mass_minus = 0.1
    p.b, p.c, p.M5 = 1.5, 0.5, 1.8
    for i in range(4):
        p.boundary_phases[2 * i] = 1.0
    h = P()
    assert L.gbf_create(name, prec, ctypes.byref(p), ctypes.byref(h)) == 0, L.gbf_last_error()
    return h

U = ctypes.create_string_buffer(64)
def update(h):
    return L.gbf_update_gauge(h, ctypes.addressof(U), 1, None)
buf = [ctypes.create_string_buffer(64) for _ in range(4)]
f = [ctypes.addressof(b) for b in buf]
def apply(h, opcode, parity=0):
    return L.gbf_apply(h, opcode, (P * 1)(f[0]), (P * 1)(f[1]), 1, parity, None)
D = ctypes.c_double * 16
one, out = D(*[1.0] * 16), D()
"""


def _run(tmp_path, body):
    from gpt_gb300 import _build

    _build.build()
    c, so = tmp_path / "fake.c", tmp_path / "libfake.so"
    c.write_text(FAKE)
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-O1", str(c), "-o", str(so)])
    env = dict(os.environ, LD_PRELOAD=str(so))
    for k in ("GBF_HOP5", "GBF_DD2"):
        env.pop(k, None)
    code = PRELUDE.format(root=ROOT, fake=str(so)) + body
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


# the four launches that start a single precision operator's vectors and hops,
# and a hop that takes another path
@pytest.mark.parametrize("call", [
    "L.gbf_axpby(h, f[2], one, None, f[0], one, f[1], 2, None)",
    "L.gbf_norm2(h, f[0], 2, out, None)",
    "L.gbf_convert(h, f[2], h64, f[0], 1.0, 2, None)",
    "L.gbf_convert(h, f[2], h64, f[0], 0.5, 2, None)",
    "apply(h, 3001)",          # one inner site per thread
    "apply(hp, 3001)",         # two inner sites per thread
    "apply(h4, 2001)",
    "apply(h64, 2001)",
])
def test_a_refused_launch_leaves_no_error_for_the_next(tmp_path, call):
    """The refused call reports its error, and neither the next call of the
    library nor another user of the runtime meets it again."""
    _run(tmp_path, f"""
h = create(b"mobius", 1, [8, 8, 8, 8], Ls=8)
hp = create(b"mobius", 1, [8, 8, 8, 8], Ls=8, n_rhs=4)
h64 = create(b"mobius", 0, [8, 8, 8, 8], Ls=8)
h4 = create(b"wilson_clover", 1, [8, 8, 8, 8])
for q in (h, hp, h64, h4):
    assert update(q) == 0, L.gbf_last_error()
    assert apply(q, 2001) == 0, L.gbf_last_error()
fake.fake_fail_launches(1)
assert ({call}) == 3
assert fake.fake_last_error() == 0
for q in (h, hp, h64, h4):
    assert apply(q, 2001) == 0, L.gbf_last_error()
assert ({call}) == 0, L.gbf_last_error()
""")


# inner sites (Ls * n_rhs) and lattice on both sides of the rule for the hops
# that read a record per 4D site: 8 inner sites, or 4 with 100,000 sites in all
@pytest.mark.parametrize("name,prec,dims,Ls,n_rhs,want", [
    ("mobius", 1, (12, 8, 10, 14), 7, 1, 0),
    ("mobius", 1, (12, 8, 10, 14), 8, 1, 1),
    ("mobius", 2, (12, 8, 10, 14), 7, 1, 0),
    ("mobius", 2, (12, 8, 10, 14), 4, 2, 1),
    ("mobius", 1, (12, 18, 18, 12), 4, 1, 0),   # 93,312
    ("mobius", 1, (14, 18, 18, 12), 4, 1, 1),   # 108,864
    ("mobius", 1, (24, 24, 24, 24), 3, 1, 0),
    ("wilson_clover", 1, (16, 16, 16, 16), 1, 4, 1),
    ("wilson_clover", 1, (16, 16, 16, 16), 1, 3, 0),
    ("mobius", 0, (12, 8, 10, 14), 12, 1, 0),
    ("mobius", 3, (12, 8, 10, 14), 12, 1, 0),
])
def test_records_are_allocated_where_the_hop_reads_them(tmp_path, name, prec, dims, Ls, n_rhs, want):
    V = dims[0] * dims[1] * dims[2] * dims[3]
    _run(tmp_path, f"""
h = create({name.encode()!r}, {prec}, {dims}, Ls={Ls}, n_rhs={n_rhs})
for i in range(2):
    assert update(h) == 0, L.gbf_last_error()
    assert fake.fake_mallocs_of({608 * V}) == {want}
    assert apply(h, 2001) == 0 and apply(h, 3002) == 0, L.gbf_last_error()
""")


def test_an_operator_works_without_memory_for_its_records(tmp_path):
    """The gauge field is taken, the operator applies (with the hop that reads
    the links), no error is left, and a later gauge field gets its records."""
    V = 8 * 8 * 8 * 8
    _run(tmp_path, f"""
h = create(b"mobius", 1, [8, 8, 8, 8], Ls=8)
fake.fake_fail_malloc({608 * V})
for i in range(2):
    assert update(h) == 0, L.gbf_last_error()
    assert fake.fake_last_error() == 0
    assert apply(h, 2001) == 0 and apply(h, 3002) == 0, L.gbf_last_error()
    assert fake.fake_mallocs_of({608 * V}) == 0
fake.fake_fail_malloc(0)
assert update(h) == 0 and apply(h, 2001) == 0, L.gbf_last_error()
assert fake.fake_mallocs_of({608 * V}) == 1
""")


def test_an_operator_without_memory_for_its_links_says_so(tmp_path):
    V = 8 * 8 * 8 * 8
    _run(tmp_path, f"""
h = create(b"mobius", 1, [8, 8, 8, 8], Ls=8)
fake.fake_fail_malloc({288 * V})
assert update(h) == 2 and b"failed" in L.gbf_last_error()
assert fake.fake_last_error() == 0
assert apply(h, 2001) == 1
""")
