/* Drives the C-ABI of the host runtime over the fake device.
 *   executor_host fail_run  early|late in out   every call of an inference that can fail does, one at a time
 *   executor_host in_place  early|late in N    one inference whose output begins N bytes into the input
 *   executor_host half      early|late in out  buffers whose first half only is page-locked, where `in` or `out` is "half"
 *   executor_host fail_load early|late - -     calls that can fail while a model is loaded do, one at a time
 *   executor_host tight     early|late - -     loads with no more device memory than the last one held, as long as that shrinks
 *   executor_host plans     early|late - -     how many convolution plans a load prepares, and its schedules
 * `in` and `out` say which memory the caller's buffers are: pageable or pinned.  Reads graph.json,
 * params.bin and input.bin of the working directory, fake::slow_images of the environment (SLOW_IMAGES), writes the bytes of the last good inference to
 * output.bin and prints "@name=value" lines.
 */
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <iterator>
#include <string>
#include <vector>
#include "cvm/c_api.h"
#include "cvm/c_api_ext.h"
#include "fake_device.h"

static std::string slurp(const char* path) {
  std::ifstream f(path, std::ios::binary);
  return std::string(std::istreambuf_iterator<char>(f), std::istreambuf_iterator<char>());
}
static char* buffer(const std::string& kind, size_t n) {
  void* p = nullptr;
  if (kind == "pinned") cudaMallocHost(&p, n);
  else p = malloc(n);
  if (kind == "half") fake::host_register(p, n / 2);
  return (char*)p;
}

int main(int argc, char** argv) {
  if (argc < 5) return 2;
  const std::string mode = argv[1], graph = slurp("graph.json"), params = slurp("params.bin"), input = slurp("input.bin");
  fake::late = std::string(argv[2]) == "late";
  auto load = [&](void** net) { return CVMAPILoadModel(graph.data(), (int)graph.size(), params.data(), (int)params.size(), net, 1, 0); };
  if (const char* n = getenv("SLOW_IMAGES")) fake::slow_images = atoi(n);
  void* net = nullptr;
  if (mode == "fail_load") {
    long failed = 0, left = 0, odd = 0;
    for (long n = 1;; n += 1 + n / 25) {
      fake::reset_calls(n);
      const int status = load(&net);
      if (status == 0) CVMAPIFreeModel(net);
      left += fake::live_objects() != 0 || fake::device_bytes != 0;
      odd += status != 0 && status != 2;
      failed += status != 0;
      if (fake::calls < n) break;
    }
    printf("@failed=%ld @left=%ld @odd=%ld\n", failed, left, odd);
    return 0;
  }
  if (mode == "plans") {
    const int status = load(&net);
    printf("@status=%d @plans=%ld\n", status, fake::conv_plans);
    char text[256] = "";
    if (status == 0 && CVMXSchedules(net, text, sizeof(text)) == 0) {
      for (char* c = text; *c; ++c) *c = *c == '\t' ? ':' : *c;
      for (char* line = strtok(text, "\n"); line; line = strtok(nullptr, "\n")) printf("@%.*s=%s\n", (int)strcspn(line, ":"), line, strchr(line, ':') + 1);
    }
    printf("@short=%d\n", status == 0 ? CVMXSchedules(net, text, 4) : -1);
    if (status == 0) CVMAPIFreeModel(net);
    return 0;
  }
  if (mode == "tight") {
    long sizes = 0, refused = 0;
    size_t least = 0;
    load(&net);
    for (size_t held = fake::device_bytes; ; held = fake::device_bytes) {
      CVMAPIFreeModel(net);
      if (held == least) break;
      ++sizes;
      least = fake::memory_limit = held;
      if (load(&net) != 0) { ++refused; break; }
    }
    printf("@sizes=%ld @refused=%ld @left=%d\n", sizes, refused, fake::live_objects() != 0);
    return 0;
  }
  if (load(&net) != 0) return 3;
  unsigned long long bytes = 0;
  CVMAPIGetOutputLength(net, &bytes);
  char* in = buffer(argv[3], input.size());
  char* out = buffer(argv[4], bytes);
  memcpy(in, input.data(), input.size());
  auto infer = [&] { return CVMAPIInference(net, in, (int)input.size(), out); };

  if (mode == "in_place") {
    free(out);
    const size_t ahead = (size_t)atoll(argv[4]);
    in = buffer(argv[3], std::max<size_t>(input.size(), ahead + bytes));
    memcpy(in, input.data(), input.size());
    out = in + ahead;
    printf("@status=%d\n", infer());
  }
  if (mode == "half") printf("@status=%d\n", infer());
  if (mode == "fail_run") {
    long failed = 0, in_flight = 0, wrong_after = 0;
    for (long n = 1;; ++n) {
      fake::reset_calls(n);
      const int status = infer();
      const bool reached = fake::calls >= n;
      const size_t pending = fake::pending();
      fake::reset_calls(0);
      if (!reached) { printf("@last_status=%d\n", status); break; }
      failed += status == 2;
      in_flight += status != 0 && pending > 0;
      memset(out, 0x55, bytes);
      if (infer() != 0 || (bytes == input.size() && memcmp(out, input.data(), bytes))) ++wrong_after;
    }
    // the same through the per-step profile, which uploads the caller's input too
    for (long n = 1;; ++n) {
      static char text[1 << 16];
      fake::reset_calls(n);
      const int status = CVMXProfileSteps(net, in, (int)input.size(), text, sizeof(text));
      const bool reached = fake::calls >= n;
      in_flight += status != 0 && fake::pending() > 0;
      fake::reset_calls(0);
      if (!reached) break;
    }
    printf("@failed=%ld @in_flight=%ld @wrong_after=%ld\n", failed, in_flight, wrong_after);
  }
  std::ofstream("output.bin", std::ios::binary).write(out, (std::streamsize)bytes);
  CVMAPIFreeModel(net);
  return 0;
}
