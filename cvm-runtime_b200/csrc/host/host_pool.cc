#include "host_pool.h"
#include <algorithm>
#include <chrono>
#include <cstring>
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

HostPool::HostPool(int helpers) {
  for (int i = 0; i < helpers; ++i) workers_.emplace_back([this] { Work(); });
}

HostPool::~HostPool() {
  {
    std::lock_guard<std::mutex> lk(mu_);
    stop_ = true;
    active_ = false;
  }
  cv_.notify_all();
  for (auto& t : workers_) t.join();
}

void HostPool::Begin() {
  {
    std::lock_guard<std::mutex> lk(mu_);
    active_ = true;
  }
  cv_.notify_all();
}

void HostPool::End() { active_.store(false, std::memory_order_release); }

void HostPool::Start(Slot slot, size_t pieces, size_t available, std::function<void(size_t)> body) {
  Job& j = jobs_[slot];
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
  Job& j = jobs_[slot];
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
  for (auto& j : jobs_)
    if (RunPiece(j)) return true;
  return false;
}

void HostPool::Work() {
  auto last = std::chrono::steady_clock::now();   // the end of the last inference seen
  bool was_active = false;
  for (;;) {
    if (active_.load(std::memory_order_acquire)) {
      was_active = true;
      if (!HelpOnce()) Relax();
      continue;
    }
    // Inferences that follow one another closely find the helpers awake: a wake-up takes about as long
    // as the first megabytes of an upload.
    const auto now = std::chrono::steady_clock::now();
    if (was_active) {
      last = now;
      was_active = false;
    }
    if (!stop_ && now - last < std::chrono::microseconds(kLingerUs)) {
      Relax();
      continue;
    }
    std::unique_lock<std::mutex> lk(mu_);
    ++asleep_;
    cv_.wait(lk, [&] { return stop_ || active_; });
    --asleep_;
    if (stop_) return;
  }
}

void HostPool::WaitPiece(Slot slot, size_t k) {
  Job& j = jobs_[slot];
  while (!j.done[k].load(std::memory_order_acquire))
    if (!RunPiece(j)) Relax();
}

void HostPool::Finish(Slot slot) {
  Job& j = jobs_[slot];
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
