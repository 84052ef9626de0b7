"""The block cache of csrc/pool.cu against a CUDA runtime made of counters: reuse,
the bound, the retries after a failed allocation, blocks of another context, a
device reset, and giving everything back.  Compiled and run on the host."""
import os
import shutil
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cuda.h>
#include <cstdio>
#include <cstdlib>
#include <map>
#include "tabi_impl.cuh"

// ---- the runtime: blocks by address, one current context, a memory limit
static unsigned long long cur = 1, next_ctx = 1;
static size_t limit = size_t(64) << 30, used = 0, largest = 0;
static int syncs = 0, objects = 0, bad = 0;
static bool sync_fails = false;
struct Live { size_t bytes; unsigned long long ctx; bool pinned; };
static std::map<char*, Live> live;
static char* top = (char*)0x1000;
static cudaError_t take(void** p, size_t n, bool pinned) {
  if (!cur) cur = ++next_ctx;
  if (used + n > limit) return cudaErrorMemoryAllocation;
  live[top] = {n, cur, pinned};
  used += n;
  *p = top;
  top += n;
  return cudaSuccess;
}
static cudaError_t drop(void* p, bool pinned) {
  auto it = live.find((char*)p);
  if (it == live.end() || it->second.pinned != pinned) { ++bad; return cudaErrorInvalidValue; }
  used -= it->second.bytes;
  live.erase(it);
  return cudaSuccess;
}
static CUresult ctx_id(CUcontext, unsigned long long* id) {
  *id = cur;
  return cur ? CUDA_SUCCESS : CUDA_ERROR_CONTEXT_IS_DESTROYED;
}
static void reset() {  // cudaDeviceReset: the context's memory is gone
  for (auto it = live.begin(); it != live.end();)
    if (it->second.ctx == cur) { used -= it->second.bytes; it = live.erase(it); } else ++it;
  objects = 0;
  cur = 0;
}
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n, false); }
cudaError_t cudaMallocHost(void** p, size_t n) { return take(p, n, true); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return take(p, n, true); }
cudaError_t cudaFree(void* p) {
  if (p) return drop(p, false);
  if (!cur) cur = ++next_ctx;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { return drop(p, true); }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaDeviceSynchronize() { ++syncs; return sync_fails ? cudaErrorUnknown : cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* a, int* b) { *a = 0; *b = -5; return cudaSuccess; }
static cudaError_t make(void** h) { ++objects; *h = (void*)(size_t)(0x77000 + objects); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return make((void**)s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) { return make((void**)s); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return make((void**)e); }
cudaError_t cudaStreamDestroy(cudaStream_t) { --objects; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { --objects; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long,
                                    cudaDriverEntryPointQueryResult* q) {
  *f = (void*)ctx_id;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
}

using namespace tabi;
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); std::exit(1); } } while (0)

int main() {
  const size_t GB = size_t(1) << 30, MB = size_t(1) << 20;
  // reuse: a block of up to twice the request, on the shelf after a wait
  MemPool::Block a = MemPool::get(3000, false);
  CHECK(a.bytes >= 3000 && live.size() == 1);
  MemPool::put(a);
  CHECK(syncs == 1 && live.size() == 1);
  MemPool::Block b = MemPool::get(2000, false);
  CHECK(b.p == a.p);
  { MemPool::Idle idle; const int s = syncs; MemPool::put(b); CHECK(syncs == s); }
  b = MemPool::get(MB, false);
  MemPool::put(b);
  CHECK(MemPool::get(1000, false).p == a.p);  // not the block of 1 MB
  MemPool::put(a);
  // a wait that fails: the block does not stay
  b = MemPool::get(8 * MB, false);
  sync_fails = true;
  MemPool::put(b);
  sync_fails = false;
  CHECK(!live.count((char*)b.p));
  // the bounds: 4 GiB, 256 MiB page-locked
  std::vector<MemPool::Block> v;
  for (int k = 0; k < 6; ++k) v.push_back(MemPool::get(GB, false));
  for (int k = 0; k < 6; ++k) v.push_back(MemPool::get(64 * MB, true));
  for (auto& x : v) MemPool::put(x);
  size_t dev = 0, pin = 0;
  for (auto& l : live) (l.second.pinned ? pin : dev) += l.second.bytes;
  CHECK(dev <= 4 * GB && dev > 2 * GB && pin == 256 * MB);
  // a failed allocation empties the shelf; then the exact size is tried
  limit = used + 512 * MB;
  b = MemPool::get(3 * GB + 1, false);
  CHECK(b.bytes > 3 * GB + 1);
  MemPool::put(b);
  MemPool::release();
  CHECK(used == 0 && live.empty());
  const size_t odd = 9 * GB + 4096;
  limit = odd;
  b = MemPool::get(odd, false);
  CHECK(b.bytes == odd);
  bool failed = false;
  try { MemPool::get(MB, false); } catch (const Error&) { failed = true; }
  CHECK(failed);
  MemPool::put(b);
  CHECK(used == 0);  // above the bound
  limit = 64 * GB;
  // under another context a block is freed, not kept, and none of the others'
  // blocks is handed out
  a = MemPool::get(MB, false);
  b = MemPool::get(MB, false);
  MemPool::put(b);
  const unsigned long long first = cur;
  cur = ++next_ctx;
  CHECK(MemPool::get(MB, false).p != b.p);
  MemPool::put(a);
  CHECK(!live.count((char*)a.p));
  MemPool::release();
  CHECK(live.count((char*)b.p));
  cur = first;
  CHECK(MemPool::get(MB, false).p == b.p);
  MemPool::put(b);
  // a large block is rounded up by little: ten of them fit where their sizes do
  MemPool::release();
  limit = used + 10 * (size_t(17) * GB + 32 * MB);
  v.clear();
  for (int k = 0; k < 10; ++k) v.push_back(MemPool::get(17 * GB + 8 * k + 1, false));
  for (auto& x : v) CHECK(x.bytes <= 17 * GB + 32 * MB);
  for (auto& x : v) MemPool::put(x);
  limit = 64 * GB;
  // bundles of streams and events: the last one back is the next one out
  HandleRes r = HandleRes::get();
  const int n = objects;
  CHECK(n == 10);
  r.put(true);
  CHECK(objects == n && HandleRes::get().stream == r.stream && objects == n);
  r.put(false);
  CHECK(objects == 0);
  for (int k = 0; k < 20; ++k) { HandleRes q; q = HandleRes::get(); q.put(true); }
  CHECK(objects == n);
  // a reset: nothing of the old context is handed out, freed or destroyed
  MemPool::Block p = MemPool::get(MB, true);
  MemPool::put(p);
  char* old = top;
  reset();
  r = HandleRes::get();
  CHECK(objects == 10 && (char*)r.h_pinned >= old);
  CHECK((char*)MemPool::get(MB, false).p >= old && (char*)MemPool::get(MB, true).p >= old);
  r.put(true);
  MemPool::release();
  CHECK(objects == 0 && bad == 0);
  std::printf("ok\n");
}
"""


def test_pool(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    csrc = os.path.join(ROOT, "tabi-pb_b200", "csrc")
    src = tmp_path / "pool_test.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "pool_test"
    r = subprocess.run([nvcc, "-x", "c++", "-std=c++17", "-O1", "-cudart", "none", "-I", csrc, "-o",
                        str(exe), str(src), os.path.join(csrc, "pool.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
