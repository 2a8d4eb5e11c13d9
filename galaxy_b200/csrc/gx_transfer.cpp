// gx_transfer.cpp -- copies between a caller's pageable arrays and the device through
// pinned staging buffers.
//
// The driver copies pageable memory through its own staging buffer on one thread; fresh
// output arrays then also take their page faults there, one after another. Here a copy
// goes in 1 MB slots: the DMA of the next ones runs while several threads move a slot
// between the staging buffer and the caller's array. Measured, us, through the driver / this
// way: inputs of 400 KB 34 / 32, 1 MB 68 / 52, 12 MB 640 / 410; outputs of 100 KB 23 / 19,
// 1 MB 90 / 49, 12 MB 720 / 336; 50 MB into new arrays 23,800 / 5,100. Arrays that are pinned
// already, and inputs below kMinIn, go directly.
//
// Making it ready costs more than a short program gains: 8 MB of pinned memory take 5 ms (4 KB
// take 2), a thread's team of 8 about 0.8 ms. So a thread's copies go directly until it has
// copied kCredit bytes (an output counts as kOutCredit at least; a larger copy is staged at
// once: its page faults alone cost more), and the last staging buffer outlives the handles,
// so that programs which make a handle a call pay once. First call of a program's only
// handle, us, through the driver / with the buffer made in each handle's first call / this
// way: 2,000 particles 767 / 5,590 / 700; 200,003 7,780 / 13,750 / 7,010. 50,000 particles in
// 8 threads of 3 calls each: 1,550 / 2,520 / 1,360.
//
// A staging buffer belongs to one call at a time. There are at most kMaxBuffers; with all of
// them in use a copy goes directly.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <new>

#include "gx_transfer.h"

namespace gx {

namespace {

constexpr size_t kSlot = size_t{1} << 20;
constexpr int kSlots = 8;
constexpr size_t kMinIn = size_t{1} << 19;
constexpr size_t kOutCredit = size_t{1} << 17;
constexpr size_t kCredit = size_t{16} << 20;
constexpr size_t kPiece = size_t{1} << 17;  // bytes a thread moves at a time
constexpr int kMaxBuffers = 4;

struct Staging {
  int device = 0;
  char* buf = nullptr;
  cudaEvent_t ev[kSlots] = {};
  bool busy[kSlots] = {};  // a DMA from the slot may be in flight (its event is recorded)
};

std::mutex g_mu;
Staging* g_idle[kMaxBuffers] = {};  // the first g_n_idle
int g_n_idle = 0;
int g_made = 0;  // idle or in use
size_t g_users = 0;
thread_local size_t t_copied = 0;

// Whether a copy is staged, counting it as so many bytes towards the thread's credit.
bool staged(size_t bytes) {
  if (t_copied <= kCredit) t_copied += std::min(bytes, kCredit + 1);
  return t_copied > kCredit;
}

void destroy(Staging* s) {
  if (!s) return;
  for (int i = 0; i < kSlots; ++i) {
    if (s->busy[i]) cudaEventSynchronize(s->ev[i]);
    if (s->ev[i]) cudaEventDestroy(s->ev[i]);
  }
  if (s->buf) cudaFreeHost(s->buf);
  delete s;
}

// A staging buffer for the current device, or null when none can be had (the caller then
// copies directly).
Staging* acquire(int device) {
  Staging* other = nullptr;  // an idle one of another device makes room
  {
    std::lock_guard<std::mutex> lk(g_mu);
    for (int i = 0; i < g_n_idle; ++i)
      if (g_idle[i]->device == device) {
        Staging* s = g_idle[i];
        g_idle[i] = g_idle[--g_n_idle];
        return s;
      }
    if (g_made == kMaxBuffers) {
      if (g_n_idle == 0) return nullptr;
      other = g_idle[--g_n_idle];
    } else {
      ++g_made;
    }
  }
  destroy(other);
  Staging* s = new (std::nothrow) Staging();
  cudaError_t e = s ? cudaSuccess : cudaErrorMemoryAllocation;
  if (s) {
    s->device = device;
    void* p = nullptr;
    e = cudaHostAlloc(&p, kSlot * kSlots, cudaHostAllocDefault);
    s->buf = static_cast<char*>(p);
  }
  for (int i = 0; i < kSlots && e == cudaSuccess; ++i) e = cudaEventCreateWithFlags(&s->ev[i], cudaEventDisableTiming);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    destroy(s);
    std::lock_guard<std::mutex> lk(g_mu);
    --g_made;
    return nullptr;
  }
  return s;
}

void release(Staging* s) {
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_users > 0 || g_n_idle == 0) {
      g_idle[g_n_idle++] = s;
      return;
    }
    --g_made;
  }
  destroy(s);
}

void move(void* dst, const void* src, size_t bytes) {
  if (bytes <= 2 * kPiece) {
    std::memcpy(dst, src, bytes);
    return;
  }
  const long long pieces = static_cast<long long>((bytes + kPiece - 1) / kPiece);
#pragma omp parallel for schedule(static) num_threads(8)
  for (long long i = 0; i < pieces; ++i) {
    const size_t o = static_cast<size_t>(i) * kPiece;
    std::memcpy(static_cast<char*>(dst) + o, static_cast<const char*>(src) + o, std::min(kPiece, bytes - o));
  }
}

bool pageable(const void* host) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

}  // namespace

void transfer_ref() {
  std::lock_guard<std::mutex> lk(g_mu);
  ++g_users;
}

void transfer_unref() {
  Staging* gone[kMaxBuffers] = {};
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_users > 0 && --g_users == 0)
      for (int i = 0; g_n_idle > 1; ++i, --g_made) gone[i] = g_idle[--g_n_idle];
  }
  for (Staging* s : gone) destroy(s);
}

cudaError_t copy_in(int device, cudaStream_t st, void* dst, const void* src, size_t bytes) {
  Staging* s = bytes >= kMinIn && pageable(src) && staged(bytes) ? acquire(device) : nullptr;
  if (!s) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
  cudaError_t e = cudaSuccess;
  int k = 0;
  for (size_t o = 0; o < bytes && e == cudaSuccess; o += kSlot, k = (k + 1) % kSlots) {
    const size_t len = std::min(kSlot, bytes - o);
    if (s->busy[k]) e = cudaEventSynchronize(s->ev[k]);
    if (e != cudaSuccess) break;
    s->busy[k] = false;
    char* slot = s->buf + static_cast<size_t>(k) * kSlot;
    move(slot, static_cast<const char*>(src) + o, len);
    e = cudaMemcpyAsync(static_cast<char*>(dst) + o, slot, len, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaEventRecord(s->ev[k], st);
    s->busy[k] = e == cudaSuccess;
  }
  release(s);
  return e;
}

namespace {

// The pieces whose bit of `which` is set, in parts of at most kSlot bytes, one after another.
struct Parts {
  const HostPiece* p;
  int count;
  unsigned which;
  int i = 0;
  size_t off = 0;
  char* dst = nullptr;
  const char* src = nullptr;
  size_t len = 0;

  bool next() {
    while (i < count && (!((which >> i) & 1u) || off >= p[i].bytes)) {
      ++i;
      off = 0;
    }
    if (i >= count) return false;
    len = std::min(kSlot, p[i].bytes - off);
    dst = static_cast<char*>(p[i].host) + off;
    src = static_cast<const char*>(p[i].dev) + off;
    off += len;
    return true;
  }
};

}  // namespace

cudaError_t copy_out(int device, cudaStream_t st, const HostPiece* pieces, int count, char* small) {
  cudaError_t e = cudaSuccess;
  unsigned which = 0;  // the pageable pieces
  size_t total = 0;
  for (int i = 0; i < count && i < 32; ++i)
    if (pieces[i].host && pieces[i].bytes && pageable(pieces[i].host)) {
      which |= 1u << i;
      total += pieces[i].bytes;
    }
  char* to = total && total <= kSmallOut ? small : nullptr;  // all of them go through `small`
  Staging* s = !to && total && staged(std::max(total, kOutCredit)) ? acquire(device) : nullptr;
  for (int i = 0; i < count && e == cudaSuccess; ++i) {
    const HostPiece& p = pieces[i];
    if (!p.host || !p.bytes) continue;
    const bool pg = i < 32 && ((which >> i) & 1u);
    if (pg && s) continue;
    e = cudaMemcpyAsync(pg && to ? to : p.host, p.dev, p.bytes, cudaMemcpyDeviceToHost, st);
    if (pg && to) to += p.bytes;
  }
  Parts in{pieces, count, s ? which : 0u}, out = in;  // issued and drained
  size_t issued = 0, drained = 0;
  bool more = in.next();
  while (e == cudaSuccess && (more || drained < issued)) {
    for (; more && issued - drained < kSlots && e == cudaSuccess; ++issued, more = in.next()) {
      const int k = static_cast<int>(issued % kSlots);
      // (stream order is not enough: the slot's last copy may be on another stream)
      if (s->busy[k]) e = cudaEventSynchronize(s->ev[k]);
      if (e == cudaSuccess) e = cudaMemcpyAsync(s->buf + k * kSlot, in.src, in.len, cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaEventRecord(s->ev[k], st);
      s->busy[k] = e == cudaSuccess;
    }
    if (e != cudaSuccess) break;
    const int k = static_cast<int>(drained % kSlots);
    e = cudaEventSynchronize(s->ev[k]);
    if (e != cudaSuccess) break;
    s->busy[k] = false;
    out.next();
    move(out.dst, s->buf + k * kSlot, out.len);
    ++drained;
  }
  if (s) release(s);
  const cudaError_t w = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = w;
  if (e == cudaSuccess && to)
    for (int i = 0; i < count && i < 32; ++i)
      if ((which >> i) & 1u) {
        std::memcpy(pieces[i].host, small, pieces[i].bytes);
        small += pieces[i].bytes;
      }
  return e;
}

}  // namespace gx
