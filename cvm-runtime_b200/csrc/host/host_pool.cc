#include "host_pool.h"
#include <algorithm>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <map>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>
#if defined(__x86_64__)
#include <emmintrin.h>
#endif

namespace cvm {

namespace {
constexpr uint64_t kCount = 0xffffffffull;
}  // namespace

void HostPool::Relax() {
#if defined(__x86_64__)
  _mm_pause();
#else
  std::this_thread::yield();
#endif
}

struct HostPool::Crew {
  std::vector<std::thread> workers;
  std::mutex mu;
  std::condition_variable cv;
  std::atomic<Desk*> desks{nullptr};
  std::atomic<int> active{0}, asleep{0};   // pools between Begin() and End(); helpers waiting for one
  std::atomic<bool> stop{false};

  explicit Crew(int helpers) {
    workers.reserve(helpers);
    try {
      for (int i = 0; i < helpers; ++i) workers.emplace_back([this] { Work(); });
    } catch (const std::system_error&) {   // (no more threads to be had: callers run what is left themselves)
    }
  }
  ~Crew() {
    {
      std::lock_guard<std::mutex> lk(mu);
      stop = true;
    }
    cv.notify_all();
    for (auto& t : workers) t.join();
    for (Desk* d = desks; d;) {
      Desk* n = d->next;
      delete d;
      d = n;
    }
  }
  Desk* TakeDesk() {
    std::lock_guard<std::mutex> lk(mu);
    for (Desk* d = desks; d; d = d->next)
      if (!d->taken) {
        d->taken = true;
        return d;
      }
    Desk* d = new Desk;
    d->taken = true;
    d->next = desks.load(std::memory_order_relaxed);
    desks.store(d, std::memory_order_release);
    return d;
  }
  // One piece of any pool's jobs, the most urgent slot first, beginning behind the pool helped last.
  bool Help(Desk** last) {
    Desk* const first = desks.load(std::memory_order_acquire);
    if (!first) return false;
    Desk* const from = *last && (*last)->next ? (*last)->next : first;
    for (int k = 0; k < kSlots; ++k) {
      Desk* d = from;
      do {
        if (d->active.load(std::memory_order_acquire) && RunPiece(d->jobs[k])) {
          *last = d;
          return true;
        }
        d = d->next ? d->next : first;
      } while (d != from);
    }
    return false;
  }
  void Work();
};

std::shared_ptr<HostPool::Crew> HostPool::crew_of(int device, int helpers) {
  static std::mutex mu;
  static std::map<int, std::weak_ptr<Crew>>& crews = *new std::map<int, std::weak_ptr<Crew>>;   // (outlives every handle)
  std::lock_guard<std::mutex> lk(mu);
  std::shared_ptr<Crew> c = crews[device].lock();
  if (!c) crews[device] = c = std::make_shared<Crew>(helpers);
  return c;
}

HostPool::HostPool(int device, int helpers) : crew_(crew_of(device, std::max(0, helpers))), desk_(crew_->TakeDesk()) {}

HostPool::~HostPool() {
  std::lock_guard<std::mutex> lk(crew_->mu);
  desk_->taken = false;
}

bool HostPool::awake() const { return crew_->asleep.load(std::memory_order_relaxed) == 0; }

void HostPool::Begin() {
  desk_->active.store(true, std::memory_order_release);
  {
    std::lock_guard<std::mutex> lk(crew_->mu);
    ++crew_->active;
  }
  crew_->cv.notify_all();
}

void HostPool::End() {
  desk_->active.store(false, std::memory_order_release);
  crew_->active.fetch_sub(1, std::memory_order_acq_rel);
}

void HostPool::Start(Slot slot, size_t pieces, size_t available, std::function<void(size_t)> body) {
  Job& j = desk_->jobs[slot];
  if (pieces > j.done_cap) {
    j.done.reset(new std::atomic<uint8_t>[pieces]);
    j.done_cap = pieces;
  }
  for (size_t k = 0; k < pieces; ++k) j.done[k].store(0, std::memory_order_relaxed);
  j.pieces = pieces;
  j.completed.store(0, std::memory_order_relaxed);
  j.body = std::move(body);
  const uint64_t gen = ((j.next.load(std::memory_order_relaxed) >> 32) + 1) << 32;
  j.next.store(gen, std::memory_order_release);
  j.avail.store(gen | available, std::memory_order_release);
}

void HostPool::Release(Slot slot, size_t available) {
  Job& j = desk_->jobs[slot];
  j.avail.store((j.next.load(std::memory_order_relaxed) & ~kCount) | available, std::memory_order_release);
}

bool HostPool::RunPiece(Job& j) {
  uint64_t n = j.next.load(std::memory_order_acquire);
  for (;;) {
    const uint64_t a = j.avail.load(std::memory_order_acquire);
    if ((n ^ a) >> 32 || (n & kCount) >= (a & kCount)) return false;
    if (j.next.compare_exchange_weak(n, n + 1, std::memory_order_acq_rel, std::memory_order_acquire)) break;
  }
  const size_t k = (size_t)(n & kCount);
  j.body(k);
  j.done[k].store(1, std::memory_order_release);
  j.completed.fetch_add(1, std::memory_order_acq_rel);
  return true;
}

bool HostPool::HelpOnce() {
  for (auto& j : desk_->jobs)
    if (RunPiece(j)) return true;
  return false;
}

void HostPool::Crew::Work() {
  constexpr int kPauses = 512;   // turns without a piece before a helper begins to yield: about 20 us
  auto last = std::chrono::steady_clock::now();   // the end of the last inference seen
  bool was_active = false;
  int idle = 0;
  Desk* helped = nullptr;
  auto turn = [&] {
    if (++idle < kPauses) Relax();
    else std::this_thread::yield();
  };
  while (!stop) {
    if (active.load(std::memory_order_acquire) > 0) {
      was_active = true;
      if (Help(&helped)) idle = 0;
      else turn();
      continue;
    }
    // Inferences that follow one another closely find the helpers awake: a wake-up takes about as long
    // as the first megabytes of an upload.
    const auto now = std::chrono::steady_clock::now();
    if (was_active) {
      last = now;
      was_active = false;
    }
    if (now - last < std::chrono::microseconds(kLingerUs)) {
      turn();
      continue;
    }
    std::unique_lock<std::mutex> lk(mu);
    ++asleep;
    cv.wait(lk, [&] { return stop || active > 0; });
    --asleep;
    idle = 0;
  }
}

void HostPool::WaitPiece(Slot slot, size_t k) {
  Job& j = desk_->jobs[slot];
  while (!j.done[k].load(std::memory_order_acquire))
    if (!RunPiece(j)) Relax();
}

void HostPool::Finish(Slot slot) {
  Job& j = desk_->jobs[slot];
  while (j.completed.load(std::memory_order_acquire) < j.pieces)
    if (!RunPiece(j)) Relax();
}

void stream_copy(char* dst, const char* src, size_t bytes) {
#if defined(__x86_64__)
  const size_t head = std::min<size_t>(bytes, (16 - ((uintptr_t)dst & 15)) & 15);
  memcpy(dst, src, head);
  dst += head; src += head; bytes -= head;
  const size_t vec = bytes & ~(size_t)63;
  for (size_t i = 0; i < vec; i += 64) {
    const __m128i a = _mm_loadu_si128((const __m128i*)(src + i)), b = _mm_loadu_si128((const __m128i*)(src + i + 16));
    const __m128i c = _mm_loadu_si128((const __m128i*)(src + i + 32)), d = _mm_loadu_si128((const __m128i*)(src + i + 48));
    _mm_stream_si128((__m128i*)(dst + i), a);
    _mm_stream_si128((__m128i*)(dst + i + 16), b);
    _mm_stream_si128((__m128i*)(dst + i + 32), c);
    _mm_stream_si128((__m128i*)(dst + i + 48), d);
  }
  _mm_sfence();
  memcpy(dst + vec, src + vec, bytes - vec);
#else
  memcpy(dst, src, bytes);
#endif
}

void stream_fill(char* dst, int byte, size_t bytes) {
#if defined(__x86_64__)
  const size_t head = std::min<size_t>(bytes, (16 - ((uintptr_t)dst & 15)) & 15);
  memset(dst, byte, head);
  dst += head; bytes -= head;
  const size_t vec = bytes & ~(size_t)63;
  const __m128i v = _mm_set1_epi8((char)byte);
  for (size_t i = 0; i < vec; i += 64) {
    _mm_stream_si128((__m128i*)(dst + i), v);
    _mm_stream_si128((__m128i*)(dst + i + 16), v);
    _mm_stream_si128((__m128i*)(dst + i + 32), v);
    _mm_stream_si128((__m128i*)(dst + i + 48), v);
  }
  _mm_sfence();
  memset(dst + vec, byte, bytes - vec);
#else
  memset(dst, byte, bytes);
#endif
}

}  // namespace cvm
