"""The pool of page-locked words behind the synchronous calls, on the CPU: csrc/host_words.h compiled
against a fake of the four CUDA runtime calls it makes, whose allocations can all be lost at once (a
device reset) and whose addresses are then used again."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG

DRIVER = r"""
#include "host_words.h"
#include <assert.h>
#include <stdlib.h>
#include <map>
#include <set>
#include <vector>
static std::map<char*, size_t> live;             // allocations of the present context
static std::multimap<size_t, char*> reusable;     // addresses that the next ones of a size get
static int frees = 0, bad_frees = 0;
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  char* m;
  auto it = reusable.find(n);
  if (it != reusable.end()) { m = it->second; reusable.erase(it); memset(m, 0, n); }
  else m = (char*)calloc(1, n);
  live[m] = n;
  *p = m;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  ++frees;
  if (live.erase((char*)p)) return cudaSuccess;
  ++bad_frees;
  return cudaErrorInvalidValue;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  a->type = cudaMemoryTypeUnregistered;
  for (auto& e : live)
    if ((const char*)p >= e.first && (const char*)p < e.first + e.second) a->type = cudaMemoryTypeHost;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
}
static void reset() {
  for (auto& e : live) { memset(e.first, 0, e.second); reusable.insert({e.second, e.first}); }
  live.clear();
}
static bool alive(const HostWords* w) {
  cudaPointerAttributes a;
  cudaPointerGetAttributes(&a, w);
  return a.type == cudaMemoryTypeHost;
}
int main() {
  {  // slots are distinct, used again, and the rest get allocations of their own
    WordPool pool;
    std::vector<WordSlot> s(70);
    std::set<HostWords*> seen;
    for (auto& x : s) { assert(pool.take(&x)); assert(alive(x.w)); seen.insert(x.w); }
    assert(seen.size() == 70 && live.size() == 8);
    HostWords* const old = s[5].w;
    pool.give(&s[5]);
    pool.give(&s[69]);
    assert(!s[5].w && live.size() == 7);
    assert(pool.take(&s[5]) && s[5].w == old);
    pool.give(&s[69]);  // given back twice: nothing
    for (auto& x : s) pool.give(&x);
    assert(live.size() == 1 && bad_frees == 0);
  }
  reset();
  reusable.clear();
  {  // a reset between: the new page gets the old one's address, the old handle's slot stays its own
    WordPool pool;
    std::vector<WordSlot> many(66);
    for (auto& x : many) assert(pool.take(&x));
    reset();
    WordSlot b, c, d;
    assert(pool.take(&b) && alive(b.w) && b.w == many[0].w);
    for (auto& x : many) pool.give(&x);  // of the lost context: neither b's slot nor its memory
    assert(pool.take(&c) && c.w != b.w && alive(c.w) && bad_frees == 0);
    pool.give(&b);
    assert(pool.take(&d) && d.w != c.w && alive(d.w));
  }
  reset();
  reusable.clear();
  {  // after a reset somebody else's buffer has the page's address: no slot lies in it
    WordPool pool;
    WordSlot a, b;
    assert(pool.take(&a));
    char* const page = (char*)a.w;
    size_t n = live[page];
    reset();
    void* other;
    cudaHostAlloc(&other, n, 0);
    assert(other == page);
    assert(pool.take(&b) && alive(b.w));
    assert((char*)b.w < page || (char*)b.w >= page + n);
    pool.give(&a);
    pool.give(&b);
    assert(live.count(page) && bad_frees == 0);
  }
  return 0;
}
"""


def test_pool_of_page_locked_words(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    inc = "/usr/local/cuda/include"
    if not cxx or not os.path.exists(os.path.join(inc, "cuda_runtime_api.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    src = tmp_path / "driver.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "driver"
    subprocess.check_call([cxx, "-std=c++17", "-O1", "-g", "-Wall", "-Werror", "-UNDEBUG", "-pthread",
                           "-I" + inc, "-I" + os.path.join(PKG, "csrc"), str(src), "-o", str(exe)])
    subprocess.check_call([str(exe)])
