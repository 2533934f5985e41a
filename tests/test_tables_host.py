"""The context's per-radius tables (csrc/tables.cpp) against a CUDA runtime of this
file's own that fails on request: a growth that fails leaves tables and radius as they
were, and a growth that succeeds never writes the tables that a launch may
still be reading."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "geopyv-dev_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
SRC = """
#include <cuda_runtime.h>
#include <cstdlib>
#include <cstring>
#include <map>
#include "internal.h"
static std::map<void *, size_t> live;
static int fail_malloc = -1, fail_copy = -1, bad_free = 0;  // calls until one fails; frees of unknown memory
cudaError_t cudaMalloc(void **p, size_t n) {
    if (fail_malloc >= 0 && fail_malloc-- == 0) { *p = nullptr; return cudaErrorMemoryAllocation; }
    *p = std::malloc(n); live[*p] = n; return cudaSuccess;
}
cudaError_t cudaFree(void *p) { if (p && !live.erase(p)) bad_free++; std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    if (fail_copy >= 0 && fail_copy-- == 0) return cudaErrorUnknown;
    std::memcpy(d, s, n); return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "made to fail"; }
namespace gpv { void set_error(const std::string &) {} int ensure_run_tables(gpv_context *, int); }
extern "C" {
void *ctx_new() { return new gpv_context(); }
void fail(int malloc_at, int copy_at) { fail_malloc = malloc_at; fail_copy = copy_at; }
int grow(gpv_context *c, int r, int runs) { return runs ? gpv::ensure_run_tables(c, r) : gpv::ensure_tables(c, r); }
int radius(gpv_context *c, int runs) { return runs ? c->run_table_radius : c->table_radius; }
// the k-th buffer of a kind of tables: its address, and its live bytes (0: not allocated)
void *buf(gpv_context *c, int runs, int k, long *bytes) {
    gpv::DevBuf *b[2][4] = {{&c->offs, &c->slots, &c->tab_off, &c->tab_n}, {&c->run_tab, nullptr, nullptr, nullptr}};
    void *p = b[runs][k] ? b[runs][k]->ptr : nullptr;
    *bytes = live.count(p) ? (long)live[p] : 0;
    return p;
}
int host_rows(gpv_context *c, int runs) { return (int)(runs ? c->h_run_n.size() : c->h_tab_n.size()); }
int frees_of_unknown() { return bad_free; }
long live_count() { return (long)live.size(); }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("tables")
    (d / "fake.cpp").write_text(SRC)
    so = str(d / "tables.so")
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC,
                    "-I", os.path.join(CUDA, "include"), "-o", so, str(d / "fake.cpp"),
                    os.path.join(CSRC, "tables.cpp"), os.path.join(CSRC, "buffers.cpp")], check=True)
    L = ct.CDLL(so)
    L.ctx_new.restype = L.buf.restype = ct.c_void_p
    L.live_count.restype = ct.c_long
    for f in (L.grow, L.radius, L.buf, L.host_rows):
        f.argtypes = [ct.c_void_p] + [ct.c_int] * {"grow": 2, "radius": 1, "buf": 2, "host_rows": 1}[f.__name__]
    L.buf.argtypes += [ct.POINTER(ct.c_long)]
    return L


def tables(L, ctx, runs):
    out = []
    for k in range(1 if runs else 4):
        n = ct.c_long()
        p = L.buf(ctx, runs, k, ct.byref(n))
        out.append((p, ct.string_at(p, n.value) if n.value else None))
    return out


@pytest.mark.parametrize("runs", [0, 1])
@pytest.mark.parametrize("what", ["malloc", "copy"])
def test_a_failed_growth_leaves_the_tables_as_they_were(lib, runs, what):
    for k in range(1 if runs else 4):
        ctx = lib.ctx_new()
        assert lib.grow(ctx, 6, runs) == 0
        before, n = tables(lib, ctx, runs), lib.live_count()
        lib.fail(k if what == "malloc" else -1, k if what == "copy" else -1)
        assert lib.grow(ctx, 30, runs) != 0
        lib.fail(-1, -1)
        assert lib.radius(ctx, runs) == 6 and lib.host_rows(ctx, runs) == 7
        assert tables(lib, ctx, runs) == before and lib.live_count() == n
        assert lib.grow(ctx, 5, runs) == 0 and tables(lib, ctx, runs) == before
        assert lib.grow(ctx, 30, runs) == 0 and lib.radius(ctx, runs) == 30
        other = lib.ctx_new()
        assert lib.grow(other, 30, runs) == 0
        assert [b for _, b in tables(lib, ctx, runs)] == [b for _, b in tables(lib, other, runs)]
    assert lib.frees_of_unknown() == 0


@pytest.mark.parametrize("runs", [0, 1])
@pytest.mark.parametrize("r0,r1", [(1, 2), (1, 3), (2, 3), (6, 7)])
def test_grown_tables_are_other_memory(lib, runs, r0, r1):
    """Tables of the smallest radii share the smallest allocation's size."""
    ctx = lib.ctx_new()
    assert lib.grow(ctx, r0, runs) == 0
    old = [p for p, _ in tables(lib, ctx, runs)]
    assert lib.grow(ctx, r1, runs) == 0
    new = [p for p, _ in tables(lib, ctx, runs)]
    assert not set(old) & set(new)


def test_run_tables_cover_the_circle(lib):
    ctx = lib.ctx_new()
    assert lib.grow(ctx, 20, 1) == 0
    t = np.frombuffer(tables(lib, ctx, 1)[0][1], np.int32)
    for r in (1, 2, 3, 13, 20):
        off, n = t[r], t[21 + r]
        run = t[42 + 2 * off:42 + 2 * (off + n)].reshape(n, 2)
        got = [(int(np.int16(w & 0xffff)), int(w >> 16) + j) for w, bits in run for j in range(4) if bits >> j & 1]
        want = [(x, y) for y in range(-r, r + 1) for x in range(-r, r + 1) if x * x + y * y <= r * r]
        assert sorted(got) == sorted(want)
