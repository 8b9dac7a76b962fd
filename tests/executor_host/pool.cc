/* The host threads that move bytes (csrc/host/host_pool.h), by themselves.
 *   pool share HANDLES   every handle runs jobs on a thread of its own; prints the most threads seen
 *   pool none            the system gives no threads (pthread_create fails)
 */
#include <dirent.h>
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <string>
#include <thread>
#include <vector>
#include "host_pool.h"

static std::atomic<bool> refuse{false};
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
  static const auto real = (int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*))dlsym(RTLD_NEXT, "pthread_create");
  return refuse ? EAGAIN : real(t, a, f, arg);
}
static int threads() {
  int n = 0;
  DIR* d = opendir("/proc/self/task");
  while (dirent* e = readdir(d)) n += e->d_name[0] != '.';
  closedir(d);
  return n;
}

// A job over each slot, pieces released in two goes, every byte checked.
static long inference(cvm::HostPool& pool, size_t pieces, unsigned char mark) {
  std::vector<unsigned char> to[3];
  cvm::HostPool::Use use;
  use.Begin(pool);
  for (int k = 0; k < 3; ++k) {
    to[k].assign(pieces * 64, 0);
    unsigned char* p = to[k].data();
    pool.Start((cvm::HostPool::Slot)k, pieces, k == 1 ? 0 : pieces, [p, mark, k](size_t i) { memset(p + i * 64, mark + k, 64); });
  }
  pool.WaitPiece(cvm::HostPool::kUpload, pieces - 1);
  pool.Release(cvm::HostPool::kDownload, pieces / 2);
  pool.HelpOnce();
  pool.ReleaseAll(cvm::HostPool::kDownload);
  for (int k = 0; k < 3; ++k) pool.Finish((cvm::HostPool::Slot)k);
  long wrong = 0;
  for (int k = 0; k < 3; ++k)
    for (unsigned char c : to[k]) wrong += c != (unsigned char)(mark + k);
  return wrong;
}

int main(int argc, char** argv) {
  std::atomic<long> wrong{0};
  if (argc > 1 && std::string(argv[1]) == "none") {
    refuse = true;
    cvm::HostPool pool(0, 5);
    for (int i = 0; i < 50; ++i) wrong += inference(pool, 9, (unsigned char)i);
    printf("@wrong=%ld @threads=%d\n", wrong.load(), threads());
    return 0;
  }
  const int handles = argc > 2 ? atoi(argv[2]) : 1, before = threads();
  std::atomic<int> most{0};
  std::unique_ptr<cvm::HostPool> stays(handles > 1 ? new cvm::HostPool(0, 5) : nullptr);
  std::vector<std::thread> callers;
  for (int h = 0; h < handles; ++h)
    callers.emplace_back([&, h] {
      for (int life = 0; life < 3; ++life) {   // (desks go from one pool to the next)
        cvm::HostPool pool(0, 5);
        for (int i = 0; i < 300; ++i) {
          wrong += inference(pool, 1 + (i * 7 + h) % 40, (unsigned char)(i + h));
          if (i % 100 == 0) {
            for (int n = threads(), m = most; n > m && !most.compare_exchange_weak(m, n);) {}
            std::this_thread::sleep_for(std::chrono::microseconds(i % 300 == 0 ? 400 : 50));
          }
        }
      }
    });
  for (auto& t : callers) t.join();
  stays.reset();
  printf("@wrong=%ld @helpers=%d @left=%d\n", wrong.load(), most.load() - before - handles, threads() - before);
  return 0;
}
