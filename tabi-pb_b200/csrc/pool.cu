// pool.cu -- process-wide cache of device and page-locked memory blocks and of
// the handles' streams and events (see MemPool and HandleRes in
// tabi_impl.cuh).
//
// A solve through a new handle spent more on allocating and freeing than on
// the solve: about 60 cudaMalloc / cudaFree pairs, page-locked staging, five
// streams and their events -- of 17.5 ms for a 1,031-atom protein of 24k faces,
// 7.5 in creating and destroying the handle and 2 in the allocations of its
// first tree.  Blocks that an object gives back stay here for the next one, up
// to a bound per context; beyond it, when an allocation fails, and when the
// program asks (tabi_release_cache), they go back to the driver.
//
// Everything is kept by the CUDA context that owns it and is only handed out or
// freed while that context is current: the id of a context is unique for the
// life of the process, so nothing of a context that cudaDeviceReset destroyed is
// met again.
#include <cuda.h>

#include "tabi_impl.cuh"

namespace tabi {

unsigned long long context_id(bool create) {
  using Query = CUresult (*)(CUcontext, unsigned long long*);
  static const Query query = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<Query>(f);
  }();
  unsigned long long id = 0;
  if (!query) return 0;
  if (query(nullptr, &id) == CUDA_SUCCESS) return id;
  // no context yet, or one that a reset destroyed: the runtime's next call makes one
  if (!create || cudaFree(nullptr) != cudaSuccess) return 0;
  return query(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

namespace {

// per context: device blocks and page-locked blocks kept, resource bundles kept
constexpr size_t kMaxDevice = size_t(4) << 30, kMaxPinned = size_t(256) << 20;
constexpr size_t kMaxRes = 16;
constexpr size_t kMaxStep = size_t(32) << 20;  // largest rounding of a block's size

thread_local int tl_idle = 0;

struct Shelf {
  std::multimap<size_t, void*> blocks;  // by size
  size_t total = 0;
};

struct Store {
  Shelf dev, pinned;
  std::vector<HandleRes> res;
};

struct Pool {
  std::mutex mu;
  std::map<unsigned long long, Store> ctx;  // by context id
};

// never destroyed: blocks that live to the end of the process go with it
Pool& pool() {
  static Pool* p = new Pool;
  return *p;
}

void trim(Shelf& sh, bool pinned) {
  for (auto& b : sh.blocks) pinned ? cudaFreeHost(b.second) : cudaFree(b.second);
  sh.blocks.clear();
  sh.total = 0;
}

}  // namespace

MemPool::Block MemPool::get(size_t bytes, bool pinned) {
  Block b;
  b.pinned = pinned;
  b.ctx = context_id(true);
  if (b.ctx) {
    Pool& P = pool();
    std::lock_guard<std::mutex> lk(P.mu);
    Store& st = P.ctx[b.ctx];
    Shelf& sh = pinned ? st.pinned : st.dev;
    auto it = sh.blocks.lower_bound(bytes);
    // at most twice the request, so that a small object does not hold a large
    // one's block
    if (it != sh.blocks.end() && it->first <= 2 * bytes + 4096) {
      b.p = it->second;
      b.bytes = it->first;
      sh.total -= b.bytes;
      sh.blocks.erase(it);
      return b;
    }
  }
  // sizes in steps of an eighth of their magnitude, so that they meet again, but of
  // at most 32 MiB: a large molecule's blocks together must not outgrow the memory
  // that their exact sizes would fit
  size_t step = 4096;
  while (16 * step < bytes && step < kMaxStep) step *= 2;
  b.bytes = (bytes + step - 1) / step * step;
  auto alloc = [&] {
    return pinned ? cudaMallocHost(&b.p, b.bytes) : cudaMalloc(&b.p, b.bytes);
  };
  cudaError_t e = alloc();
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    if (b.ctx) {
      Pool& P = pool();
      std::lock_guard<std::mutex> lk(P.mu);
      Store& st = P.ctx[b.ctx];
      trim(pinned ? st.pinned : st.dev, pinned);
    }
    e = alloc();
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      b.bytes = bytes;
      e = alloc();
    }
  }
  TABI_CUDA(e);
  return b;
}

void MemPool::put(Block b) {
  if (!b.p) return;
  // under another context the owner's work is not known to be done
  bool keep = b.ctx != 0 && b.ctx == context_id(false);
  if (keep && !b.pinned && tl_idle == 0) keep = cudaDeviceSynchronize() == cudaSuccess;
  if (keep) {
    Pool& P = pool();
    std::lock_guard<std::mutex> lk(P.mu);
    Store& st = P.ctx[b.ctx];
    Shelf& sh = b.pinned ? st.pinned : st.dev;
    if (sh.total + b.bytes <= (b.pinned ? kMaxPinned : kMaxDevice)) {
      sh.blocks.emplace(b.bytes, b.p);
      sh.total += b.bytes;
      return;
    }
  }
  b.pinned ? cudaFreeHost(b.p) : cudaFree(b.p);
}

void MemPool::release() {
  Store st;
  {
    Pool& P = pool();
    std::lock_guard<std::mutex> lk(P.mu);
    auto it = P.ctx.find(context_id(false));
    if (it == P.ctx.end()) return;
    std::swap(st, it->second);
    P.ctx.erase(it);
  }
  trim(st.dev, false);
  trim(st.pinned, true);
  for (HandleRes& r : st.res) r.destroy();
}

MemPool::Idle::Idle() {
  ok = cudaDeviceSynchronize() == cudaSuccess;
  if (ok) ++tl_idle;
}
MemPool::Idle::~Idle() {
  if (ok) --tl_idle;
}

HandleRes HandleRes::get() {
  const unsigned long long id = context_id(true);
  if (id) {
    Pool& P = pool();
    std::lock_guard<std::mutex> lk(P.mu);
    std::vector<HandleRes>& v = P.ctx[id].res;
    if (!v.empty()) {
      HandleRes r = v.back();
      v.pop_back();
      return r;
    }
  }
  HandleRes r;
  r.ctx = id;
  try {
    int prio_lo = 0, prio_hi = 0;
    TABI_CUDA(cudaDeviceGetStreamPriorityRange(&prio_lo, &prio_hi));
    const int prio_mid = (prio_lo + prio_hi) / 2;
    TABI_CUDA(cudaStreamCreateWithFlags(&r.stream, cudaStreamNonBlocking));
    TABI_CUDA(cudaStreamCreateWithFlags(&r.side, cudaStreamNonBlocking));
    TABI_CUDA(cudaStreamCreateWithPriority(&r.lu_hi, cudaStreamNonBlocking, prio_hi));
    TABI_CUDA(cudaStreamCreateWithPriority(&r.aux, cudaStreamNonBlocking, prio_mid));
    TABI_CUDA(cudaStreamCreateWithPriority(&r.lu_small, cudaStreamNonBlocking, prio_mid));
    for (cudaEvent_t* e : {&r.ev_fork, &r.ev_join, &r.ev_la, &r.ev_rest, &r.ev_lu_join})
      TABI_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
    TABI_CUDA(cudaMallocHost(&r.h_pinned, sizeof(double) * 256));
  } catch (...) {
    r.destroy();
    throw;
  }
  return r;
}

void HandleRes::put(bool idle) {
  if (idle && stream && h_pinned && ctx != 0 && ctx == context_id(false)) {
    Pool& P = pool();
    std::lock_guard<std::mutex> lk(P.mu);
    std::vector<HandleRes>& v = P.ctx[ctx].res;
    if (v.size() < kMaxRes) {
      v.push_back(*this);
      return;
    }
  }
  destroy();
}

void HandleRes::destroy() {
  for (cudaStream_t s : {stream, side, lu_hi, aux, lu_small})
    if (s) cudaStreamDestroy(s);
  for (cudaEvent_t e : {ev_fork, ev_join, ev_la, ev_rest, ev_lu_join})
    if (e) cudaEventDestroy(e);
  if (h_pinned) cudaFreeHost(h_pinned);
}

}  // namespace tabi
