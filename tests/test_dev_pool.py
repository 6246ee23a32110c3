"""The pool of plans' device memory (csrc/dev_pool.h), compiled as plain C++
over a stand-in for the CUDA runtime: what is handed out again and when, what
happens where the device cannot be waited for, and at the ends of device and
host memory."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SOURCE = r"""
#include "dev_pool.h"
#include <cstdio>
#include <cstdlib>
#include <map>
#include <thread>
#include <vector>

// the runtime: `room` bytes of device memory, waits that can be refused, operator new that can run out
static size_t room = size_t(1) << 40;
static bool refuse_wait = false;
static int no_new_after = -1;
static std::map<void*, size_t>& live() { static std::map<void*, size_t> m; return m; }
static std::mutex rt;
static char next_block[1 << 16];
static size_t next_at = 0;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  std::lock_guard<std::mutex> l(rt);
  if (n > room) return cudaErrorMemoryAllocation;
  room -= n;
  *p = &next_block[next_at++];
  const int keep = no_new_after;
  no_new_after = -1;
  live()[*p] = n;
  no_new_after = keep;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::lock_guard<std::mutex> l(rt);
  if (!p) return cudaSuccess;
  if (!live().count(p)) { std::puts("freed twice"); std::exit(2); }
  room += live()[p];
  live().erase(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return refuse_wait ? cudaErrorStreamCaptureUnsupported : cudaSuccess; }
}
void* operator new(size_t n) {
  if (no_new_after == 0) throw std::bad_alloc();
  if (no_new_after > 0) --no_new_after;
  return std::malloc(n);
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

static int reuse() {
  DevPool pool(0);
  void *a, *b, *c, *d;
  CHECK(pool.get(&a, 100000) == cudaSuccess && pool.get(&b, 300000) == cudaSuccess && a != b);
  pool.give({a, nullptr, b});
  CHECK(pool.get(&c, 99000) == cudaSuccess && c == a);    // the smallest that fits
  CHECK(pool.get(&d, 140000) == cudaSuccess && d != b);   // 300,000 would waste more than half
  CHECK(pool.get(&a, 299000) == cudaSuccess && a == b);
  pool.put(nullptr);
  pool.put(c);
  CHECK(pool.get(&b, 100000) == cudaSuccess && b == c);
  pool.give({a, b, d});
  return 0;
}
static int aside() {  // a block that may be in use
  DevPool pool(0);
  void *a, *b, *c;
  CHECK(pool.get(&a, 1000) == cudaSuccess);
  refuse_wait = true;
  pool.give({a});
  CHECK(pool.get(&b, 1000) == cudaSuccess && b != a);
  refuse_wait = false;
  CHECK(pool.get(&c, 1000) == cudaSuccess && c != a);  // no wait has succeeded yet
  pool.give({b});                                      // now both are done with
  void *x, *y;
  CHECK(pool.get(&x, 1000) == cudaSuccess && pool.get(&y, 1000) == cudaSuccess);
  CHECK((x == a && y == b) || (x == b && y == a));
  refuse_wait = true;
  pool.give({x});  // left aside when the pool goes
  refuse_wait = false;
  pool.give({y, c});
  return 0;
}
static int limit() {
  DevPool pool(0);
  void *a, *b;
  CHECK(pool.get(&a, DevPool::kLimit) == cudaSuccess && pool.get(&b, 4096) == cudaSuccess);
  pool.give({a});
  CHECK(live().size() == 2);
  pool.give({b});  // beyond the limit
  CHECK(live().size() == 1);
  return 0;
}
static int full() {  // device memory runs out: what the pool holds goes first
  DevPool pool(0);
  void *a, *b;
  CHECK(pool.get(&a, 1 << 20) == cudaSuccess);
  pool.give({a});
  room = 1 << 19;
  CHECK(pool.get(&b, 3 << 18) == cudaSuccess);
  pool.give({b});
  void* c;
  CHECK(room < (3 << 18) && pool.outside(&c, 5 << 18) == cudaSuccess);
  CHECK(pool.outside(&b, 1 << 30) == cudaErrorMemoryAllocation && pool.get(&b, 1 << 30) == cudaErrorMemoryAllocation);
  cudaFree(c);
  room = size_t(1) << 40;
  return 0;
}
static int host_full() {  // host memory runs out
  DevPool pool(0);
  void* a = nullptr;
  no_new_after = 0;
  const cudaError_t e = pool.get(&a, 4096);
  no_new_after = -1;
  CHECK(e == cudaErrorMemoryAllocation && live().empty());
  CHECK(pool.get(&a, 4096) == cudaSuccess);
  no_new_after = 0;
  pool.give({a});
  no_new_after = -1;
  void* b;
  CHECK(pool.get(&b, 4096) == cudaSuccess && a == b);
  pool.give({b});
  return 0;
}
static int threads() {
  DevPool pool(0);
  std::vector<std::thread> ts;
  bool bad[8] = {};
  for (int t = 0; t < 8; ++t)
    ts.emplace_back([&, t] {
      for (int i = 0; i < 2000; ++i) {
        void *a = nullptr, *b = nullptr;
        if (pool.get(&a, 1000 + t) != cudaSuccess || pool.get(&b, 70000) != cudaSuccess || a == b) bad[t] = true;
        if (i % 3) pool.give({a, b}); else { pool.put(a); pool.give({b}); }
      }
    });
  for (auto& t : ts) t.join();
  for (bool b : bad) CHECK(!b);
  return 0;
}
int main(int, char** v) {
  const std::string_view w(v[1]);
  const int rc = w == "reuse" ? reuse() : w == "aside" ? aside() : w == "limit" ? limit() : w == "full" ? full()
               : w == "host_full" ? host_full() : threads();
  if (!rc && !live().empty()) { std::puts("left behind"); return 3; }  // the pool is gone by now
  return rc;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("pool")
    src, exe = d / "p.cpp", d / "p"
    src.write_text(SOURCE.replace('#include <cstdio>', '#include <cstdio>\n#include <string_view>', 1))
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", f"-I{CUDA}/include",
                    "-I" + os.path.join(ROOT, "gitm_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("what", ["reuse", "aside", "limit", "full", "host_full", "threads"])
def test_pool(program, what):
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
