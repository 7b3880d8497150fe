"""The device-block cache of a context (csrc/fl_blocks.h) over a fake device
heap: no GPU, the header compiled with the host compiler."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fiber-raman-suppression_b200", "csrc")

HARNESS = r"""
#include "fl_blocks.h"
#include <cstdio>
#include <cstdlib>
#include <map>
using fl::BlockCache;
static const size_t MB = size_t(1) << 20;
static std::map<char*, size_t> heap;      // the fake device's blocks
static size_t in_use = 0, capacity = size_t(1) << 40;
static int syncs = 0;
static bool stream_dead = false, stream_busy = false;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
    if (in_use + n > capacity) return cudaErrorMemoryAllocation;
    char* q = (char*)malloc(1);
    heap[q] = n;
    in_use += n;
    *p = q;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    auto it = heap.find((char*)p);
    if (it == heap.end()) { puts("free of an unknown block"); exit(1); }
    in_use -= it->second;
    heap.erase(it);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    if (stream_dead) { puts("a destroyed stream was used"); exit(1); }
    syncs++;
    if (stream_busy) return cudaErrorNotReady;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
}
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

static int reuse() {                      // handed on, after one wait for the stream
    BlockCache c;
    void *a, *b, *d;
    CHECK(!c.alloc(&a, 3 * MB) && !c.alloc(&d, 5 * MB));
    c.release(a);
    c.release(d);
    CHECK(syncs == 0 && in_use == 8 * MB);
    CHECK(!c.alloc(&b, 2 * MB) && b == a && syncs == 1);
    CHECK(!c.alloc(&a, 5 * MB) && a == d && syncs == 1);
    CHECK(!c.alloc(&d, 1 * MB) && in_use == 9 * MB);
    c.release(b);
    CHECK(!c.alloc(&b, 1 * MB) && in_use == 10 * MB);   // (no more than twice the request)
    c.close();
    CHECK(in_use == 7 * MB);
    c.release(a); c.release(b); c.release(d); c.release(nullptr);
    CHECK(in_use == 0);
    return 0;
}
static int stream_gone() {                // the caller's stream ended before its objects
    BlockCache c;
    c.set_stream((cudaStream_t)1);
    void *a, *b;
    CHECK(!c.alloc(&a, MB));
    stream_dead = true;
    c.release(a);
    c.set_stream((cudaStream_t)2);        // (what was queued on the old one has run)
    CHECK(!c.alloc(&b, MB) && b == a);
    c.release(b);
    c.close();
    CHECK(in_use == 0);
    return 0;
}
static int busy() {                       // a wait that fails: a block of its own
    BlockCache c;
    void *a, *b;
    CHECK(!c.alloc(&a, MB));
    c.release(a);
    stream_busy = true;
    CHECK(!c.alloc(&b, MB) && b != a && in_use == 2 * MB);
    c.release(b);
    c.close();
    CHECK(in_use == 0);
    return 0;
}
static int memory_full() {                // spare blocks go before an allocation fails
    auto c = std::make_shared<BlockCache>();
    auto other = std::make_shared<BlockCache>();
    other->close();
    other->set_lender(c);
    capacity = 100 * MB;
    void *a, *b;
    CHECK(!c->alloc(&a, 60 * MB));
    c->release(a);
    CHECK(in_use == 60 * MB);
    CHECK(!other->alloc(&b, 80 * MB) && in_use == 80 * MB);
    CHECK(other->alloc(&a, 30 * MB) == cudaErrorMemoryAllocation);
    other->release(b);
    CHECK(in_use == 0);                   // (that one keeps nothing)
    CHECK(!c->alloc(&a, 60 * MB));
    c->release(a);
    CHECK(!c->alloc(&a, 90 * MB) && in_use == 90 * MB);
    c->release(a);
    c->close();
    CHECK(in_use == 0);
    return 0;
}
static int bounds() {                     // kKeep, and a context's budget
    void* p[8];
    BlockCache c;
    for (int i = 0; i < 8; i++) CHECK(!c.alloc(&p[i], 60 * MB));
    for (int i = 0; i < 8; i++) c.release(p[i]);
    CHECK(in_use <= BlockCache::kKeep && in_use >= 200 * MB);
    CHECK(!c.alloc(&p[0], 200 * MB));     // half of kKeep and more: not kept
    c.release(p[0]);
    CHECK(in_use <= BlockCache::kKeep);
    c.close();
    CHECK(in_use == 0);
    BlockCache s(40 * MB);
    for (int i = 0; i < 4; i++) CHECK(!s.alloc(&p[i], 20 * MB));
    for (int i = 0; i < 4; i++) s.release(p[i]);
    CHECK(in_use <= 40 * MB && in_use >= 20 * MB);
    CHECK(!s.alloc(&p[0], 30 * MB) && in_use <= 40 * MB);
    s.release(p[0]);
    CHECK(!s.alloc(&p[0], 16 * MB) && in_use <= 40 * MB);
    s.release(p[0]);
    s.close();
    CHECK(in_use == 0);
    return 0;
}
int main(int argc, char** argv) {
    const std::string t = argv[1];
    return t == "reuse" ? reuse() : t == "stream_gone" ? stream_gone() : t == "busy" ? busy()
         : t == "memory_full" ? memory_full() : bounds();
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not (os.path.exists(os.path.join(inc, "cuda_runtime_api.h")) and shutil.which("g++")):
        pytest.skip("no host compiler or CUDA headers")
    d = tmp_path_factory.mktemp("blocks")
    (d / "t.cpp").write_text("#include <string>\n" + HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", f"-I{inc}",
                    str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("what", ["reuse", "stream_gone", "busy", "memory_full", "bounds"])
def test_block_cache(harness, what):
    r = subprocess.run([harness, what], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
