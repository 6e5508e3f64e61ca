"""csrc/device_pool.cuh against a fake CUDA runtime with a small memory: no GPU needed."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gllm-kernels_b200", "csrc")

FAKE = r"""
#pragma once
#include <cstddef>
#include <cstdlib>
#include <map>
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2 };
struct Fake { std::map<void *, size_t> live; size_t used = 0, room = (size_t)512 << 20; int mallocs = 0, waits = 0; };
inline Fake &fake() { static Fake f; return f; }
inline cudaError_t cudaMalloc(void **p, size_t n) {
    Fake &f = fake();
    if (f.used + n > f.room) return cudaErrorMemoryAllocation;
    *p = std::malloc(1);
    f.live[*p] = n; f.used += n; f.mallocs++;
    return cudaSuccess;
}
inline cudaError_t cudaFree(void *p) { Fake &f = fake(); f.used -= f.live.at(p); f.live.erase(p); std::free(p); return cudaSuccess; }
inline cudaError_t cudaDeviceSynchronize() { fake().waits++; return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
"""


def run(tmp_path, body):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "t.cpp").write_text(
        '#include "device_pool.cuh"\n#include <cstdio>\nusing namespace gllmk;\n'
        '#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\\n", __LINE__, #c); return 1; } } while (0)\n'
        '#define TAKE(d, n, p, w) pool_take(d, n, p, true, w)\n'
        'constexpr size_t MB = (size_t)1 << 20;\n'
        'int main() {\n' + body + '\nreturn 0;\n}\n')
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", CSRC, "-x", "c++", str(tmp_path / "t.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_an_allocation_has_the_size_that_was_asked_for(tmp_path):
    """Model weights are allocated once and kept: 33.9 MB are 33.9 MB."""
    run(tmp_path, r"""
    pool_of(0).contexts = 1;
    for (size_t want : {(size_t)33882112, (size_t)51380240, (size_t)100, (size_t)90 * MB + 16}) {
        size_t n = want; void *p; bool waited = false;
        const size_t before = fake().used;
        CHECK(TAKE(0, &n, &p, &waited) == cudaSuccess && n == want && !waited && fake().used - before == want);
    }""")


def test_a_freed_buffer_serves_requests_of_about_its_size(tmp_path):
    run(tmp_path, r"""
    pool_of(0).contexts = 1;
    size_t n = 9 * MB; void *p, *q; bool waited = false;
    CHECK(TAKE(0, &n, &p, &waited) == cudaSuccess);
    pool_put(0, p, n);
    n = 10 * MB;  // too small for this
    CHECK(TAKE(0, &n, &q, &waited) == cudaSuccess && q != p && !waited);
    n = 7 * MB;   // more than an eighth larger than this
    CHECK(TAKE(0, &n, &q, &waited) == cudaSuccess && q != p && n == 7 * MB && !waited);
    n = 8 * MB;   // an eighth larger: taken, after the device has been waited for, at its own size
    CHECK(TAKE(0, &n, &q, &waited) == cudaSuccess && q == p && n == 9 * MB && waited && fake().waits == 1);
    pool_put(0, q, n);
    // the closest of several, and small ones within 64 KB
    void *a, *b; size_t na = 8 * MB + 4096, nb = 4096;
    CHECK(cudaMalloc(&a, na) == cudaSuccess && cudaMalloc(&b, 65536) == cudaSuccess);
    pool_put(0, a, na); pool_put(0, b, 65536);
    n = 8 * MB;
    CHECK(TAKE(0, &n, &q, &waited) == cudaSuccess && q == a && n == na);
    CHECK(TAKE(0, &nb, &q, &waited) == cudaSuccess && q == b && nb == 65536);
    // bounded: at most 128 MB, the oldest go first; none beyond 64 MB, none without a context
    for (int i = 0; i < 5; i++) { CHECK(cudaMalloc(&a, 40 * MB) == cudaSuccess); pool_put(0, a, 40 * MB); CHECK(pool_of(0).held <= POOL_MAX_BYTES); }
    CHECK(cudaMalloc(&a, 65 * MB) == cudaSuccess);
    const size_t used = fake().used;
    pool_put(0, a, 65 * MB);
    CHECK(fake().used == used - 65 * MB);
    pool_trim(0);
    CHECK(pool_of(0).held == 0 && pool_of(0).blocks.empty());""")


def test_an_upload_from_the_host_takes_no_freed_buffer(tmp_path):
    """It would have to wait for the device, which no thread may do while another one captures a stream."""
    run(tmp_path, r"""
    pool_of(0).contexts = 1;
    size_t n = 9 * MB; void *p, *q; bool waited = false;
    CHECK(pool_take(0, &n, &p, true, &waited) == cudaSuccess);
    pool_put(0, p, n);
    CHECK(pool_take(0, &n, &q, false, &waited) == cudaSuccess && q != p && !waited && fake().waits == 0);""")


def test_any_allocation_may_claim_the_idle_buffers(tmp_path):
    run(tmp_path, r"""
    pool_of(0).contexts = 1;
    void *p, *q;
    for (int i = 0; i < 3; i++) { CHECK(cudaMalloc(&p, 40 * MB) == cudaSuccess); pool_put(0, p, 40 * MB); }
    CHECK(pool_of(0).held == 120 * MB);
    CHECK(device_malloc(0, &p, 380 * MB) == cudaSuccess && pool_of(0).held == 120 * MB);  // fits beside them
    CHECK(device_malloc(0, &q, 100 * MB) == cudaSuccess && pool_of(0).held == 0);         // only without them
    CHECK(device_malloc(0, &p, 512 * MB) == cudaErrorMemoryAllocation);""")


def test_the_library_allocates_device_memory_in_one_place():
    """cudaMalloc elsewhere would fail while idle weight buffers could be given back."""
    import re
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")) and name != "device_pool.cuh":
            with open(os.path.join(CSRC, name)) as f:
                code = re.sub(r'//[^\n]*|"[^"\n]*"', "", f.read())
                assert not re.search(r"\bcudaMalloc\s*\(", code), name
