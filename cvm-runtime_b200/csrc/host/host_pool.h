// A few host threads that move bytes for the calling thread of an inference: a pageable caller
// buffer into the page-locked staging buffer, downloaded pieces into the caller's output buffer,
// constant fills.  Each of these is a job cut into pieces; a piece is a call of the job's body.
//
// A HostPool is what one handle has of them: its jobs.  The threads belong to a crew that all handles of a
// device share, started with the first of them and ended with the last: three handles on one GPU keep
// five helpers busy, not fifteen.
//
// The helpers sleep between inferences that are more than a fifth of a millisecond apart.  Begin() wakes
// them, and until End() they spin over the jobs, lowest slot first, so that a job that starts while others
// run is picked up without a wake-up (tens of microseconds, more than many of these jobs take); after some
// twenty microseconds without a piece they offer their core to other threads between two looks.  The caller
// helps with every job it waits for.
#pragma once
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <functional>
#include <memory>

namespace cvm {

class HostPool {
 public:
  enum Slot { kUpload = 0, kDownload = 1, kFill = 2, kSlots = 3 };   // in order of urgency

  // `device` names the crew; `helpers` is how many threads it has if it does not exist yet (fewer where the
  // system gives no more, none is fine).
  HostPool(int device, int helpers);
  ~HostPool();
  HostPool(const HostPool&) = delete;
  HostPool& operator=(const HostPool&) = delete;

  void Begin();
  void End();
  // Starts a job of `pieces` calls body(k).  The slot's previous job must have finished.  The first
  // `available` pieces may run at once, the others when Release() says so.
  void Start(Slot slot, size_t pieces, size_t available, std::function<void(size_t)> body);
  void Release(Slot slot, size_t available);
  void ReleaseAll(Slot slot) { Release(slot, desk_->jobs[slot].pieces); }
  // Waits until piece k has run, running pieces of this job meanwhile.
  void WaitPiece(Slot slot, size_t k);
  // Waits until the whole job has run.
  void Finish(Slot slot);
  static void Relax();   // one turn of a spin
  // Runs one piece of any job, if one is free; false if there is none.
  bool HelpOnce();

  // Helpers at work, until it goes out of scope: whatever way that comes about, all jobs have run by then
  // and none touches the buffers of their bodies afterwards.
  struct Use {
    HostPool* p = nullptr;
    Use() = default;
    Use(const Use&) = delete;
    Use& operator=(const Use&) = delete;
    void Begin(HostPool& pool) {
      if (p) return;   // (at work already)
      p = &pool;
      p->Begin();
    }
    ~Use() {
      if (!p) return;
      for (int k = 0; k < kSlots; ++k) {
        p->ReleaseAll((Slot)k);   // (pieces that an error kept back)
        p->Finish((Slot)k);
      }
      p->End();
    }
  };

  static constexpr int kLingerUs = 200;
  bool awake() const;   // Begin() needs no wake-up

 private:
  // (a cache line or more to itself: helpers poll all of them)
  struct alignas(64) Job {
    // (generation << 32 | count): a claim is a compare-exchange of the whole word against `avail` of
    // the same generation, so a helper that looked at the slot's previous job cannot take a
    // piece the present one does not have.
    std::atomic<uint64_t> next{0}, avail{0};
    std::function<void(size_t)> body;
    size_t pieces = 0;
    std::unique_ptr<std::atomic<uint8_t>[]> done;
    size_t done_cap = 0;
    std::atomic<size_t> completed{0};
  };
  // The jobs of one pool.  The crew never frees a desk while its threads run, so that they may look at any at
  // any time; a desk whose pool is gone has no pieces to claim and goes to the next pool.
  struct Desk {
    Job jobs[kSlots];
    alignas(64) std::atomic<bool> active{false};
    bool taken = false;
    Desk* next = nullptr;
  };
  struct Crew;
  static std::shared_ptr<Crew> crew_of(int device, int helpers);
  static bool RunPiece(Job& j);

  std::shared_ptr<Crew> crew_;
  Desk* desk_;
};

// memcpy with stores that bypass the cache: for destinations the CPU does not read soon (the
// staging buffer the copy engine reads, a large output).
void stream_copy(char* dst, const char* src, size_t bytes);
void stream_fill(char* dst, int byte, size_t bytes);   // memset the same way

}  // namespace cvm
