// Device executor: lowers a validated Graph into a static list of kernel launches on one GPU and
// replays it per inference.
//
// The reference executor (CvmRuntime::SetupStorage / SetupOpExecs / Run,
// src/runtime/graph_runtime.cc:576-698, :61-68) binds one int32 buffer per entry and runs one
// operator body per node.  This one keeps the node-by-node semantics but chooses, at load time,
//   - a storage type per entry: int8 where every value is provably within [-127, 127], else int32;
//   - a physical layout: 4-D entries are held channels-last (NHWC), everything else row-major;
//   - fusion: chains of element-wise successors with a single consumer are folded into the
//     producing kernel (conv2d / dense / reduce / element-wise), so their int32 intermediates are
//     never written;
//   - pre-packed int8 weights (OIHW -> OHWI) and TMA tensor maps for the tensor-core convolutions;
//   - CUDA graphs: one of every step and the way of the heads to the host, behind a kernel that fetches
//     the staging buffer where the input is small; and, for batches that upload while they compute,
//     one per part of the batch over the leading steps, launched when the part is on the device
//     (Schedule).  Where the cut lies is timed at load, for inputs in page-locked, pageable and
//     device memory separately.
// The result is written into page-locked memory by a kernel (small heads), or leaves in pieces that host
// threads (HostPool) move on, part by part of the batch where the whole graph runs that way.
// There is no CPU fallback: every step is a CUDA kernel from this library.
#pragma once
#include <cuda_runtime.h>
#include <chrono>
#include <functional>
#include <memory>
#include <string>
#include <vector>
#include "cvmk_kernels.h"
#include "graph.h"
#include "host_pool.h"

namespace cvm {

struct DevBuf {
  Shape shape;          // logical shape
  int dtype = CVMK_I32; // CVMK_I8 / CVMK_I32
  bool nhwc = false;    // 4-D tensor stored as N,H,W,C
  void* ptr = nullptr;
  size_t bytes() const { return (size_t)shape_size(shape) * dtype; }
};

struct Step {
  std::string label;
  std::function<int(cudaStream_t)> launch;
  // The same operator on one part of the batch each (empty when the step cannot be cut along the
  // batch): the leading steps of an inference run part by part while later parts upload.
  std::vector<std::function<int(cudaStream_t)>> chunk;
  int64_t images = 0;        // of the batch that `chunk` cuts
  bool from_input = false;   // reads the uploaded bytes and nothing else of the batch
};

struct HeadOut {
  Shape shape;
  int dtype;
  void* dev = nullptr;       // canonical row-major copy on the device
  void* host = nullptr;      // pinned
  size_t bytes = 0;
  // The output of non_max_suppression with a limit on its rows: of every image only the first
  // live_bytes can hold anything but -1, so only those are downloaded (0: the whole tensor is).
  size_t images = 1, live_bytes = 0;
  const int32_t* valid_count = nullptr;   // device, [images]: an image with none ends the operator's loop
};

class Executor {
 public:
  // `plain_elem_bytes`: when not 0, the caller wants a single head's elements as they are, this many
  // bytes each, and hands Run() the buffer for them (see delivers_output()).
  Executor(const Graph& g, int device_id, int plain_elem_bytes);
  ~Executor();
  // Runs one inference.  `input` holds the `data` tensor in API form (int8 or int32, row-major).
  // If delivers_output(), the head's bytes are in `out` on return; otherwise heads()[k].host holds
  // head k (row-major, heads()[k].dtype).
  void Run(const void* input, size_t input_bytes, char* out);
  bool delivers_output() const { return plain_; }
  const std::vector<HeadOut>& heads() const { return heads_; }
  size_t num_steps() const { return steps_.size(); }
  size_t device_bytes() const { return device_bytes_; }
  void activation_bytes(unsigned long long* buffers, unsigned long long* physical) const {
    *buffers = 0;
    for (const auto& a : act_) *buffers += a.va_size;
    *physical = 0;
    for (const auto& b : phys_) *physical += b.size;
  }
  // Per-step device times of one eager pass (label, milliseconds); used by the profiling table.
  std::vector<std::pair<std::string, float>> ProfileOnce(const void* input, size_t input_bytes);
  // Replays only the kernels (input already in device memory, no upload / download) `iters`
  // times and returns the device time in milliseconds measured with CUDA events on the stream.
  float ReplayDevice(int iters);
  // The schedules chosen at load (CVMXSchedules).
  std::string DescribeSchedules() const;
  // Writes `code` into the device status word the kernels report their expired waits in.
  void SetStatusWord(int code);

 private:
  struct Impl;
  const Graph& g_;
  int device_;
  cudaStream_t stream_ = nullptr;
  std::vector<Step> steps_;
  enum class Source { kDirect, kSmall, kPool };   // read where it lies; staged by the caller; staged by the pool
  static constexpr size_t kSmallInput = (size_t)1 << 20, kSmallDirect = (size_t)1 << 18;
  // A small input (or head) of at least kSmallShare is copied together with the pool's helpers if they are
  // awake (547 KB 166 -> 150 us a call, 150 KB 224.4 -> 222.8); asleep, waking them costs more than that.
  static constexpr size_t kSmallShare = (size_t)64 << 10, kSmallPiece = (size_t)32 << 10;
  static constexpr size_t kStagePiece = (size_t)256 << 10, kDownloadPiece = (size_t)1 << 20;
  // An inference: the first `prefix` steps part by part, one graph per part of the batch, each launched
  // when its part of the input is on the device; the last part's graph goes on with the rest of the
  // steps and the delivery of the heads.  Without a prefix: one graph.
  struct DropGraph {
    void operator()(cudaGraphExec_t g) const { cudaGraphExecDestroy(g); }
  };
  using GraphExec = std::unique_ptr<CUgraphExec_st, DropGraph>;
  struct Schedule {
    size_t prefix = 0;
    int cut = 0;                            // which parts (kCuts)
    std::vector<GraphExec> graphs;
  };
  // How long the prefix should be depends on how fast the input arrives: chosen at load by timing
  // inferences, once from page-locked memory (read by the copy engine where it lies) and once from
  // pageable memory (staged by host threads first).  prefix_max_ bounds it (the memory planner keeps
  // everything those steps touch live together).
  Schedule from_pinned_, from_pageable_;
  Schedule from_device_;   // an input in device memory: the whole graph, unless the head's parts can leave early
  GraphExec graph_whole_;    // every step: the input is on the device already
  GraphExec graph_staged_;   // the same behind a kernel that fetches the staging buffer (small inputs)
  size_t prefix_max_ = 0;
  Schedule MakeSchedule(size_t prefix, int cut);
  void Load(int plain_elem_bytes);
  void Release();
  GraphExec Capture(const std::function<void()>& enqueue);
  void ChooseSchedules();
  void Launch(const void* input, Source src, const Schedule& how, char* head, bool early);
  static bool IsDirect(const void* p, size_t bytes);
  static bool IsDevice(const void* input);
  std::vector<size_t> range_end_;   // input bytes up to the end of each range of images that steps are prepared for
  std::vector<size_t> head_range_end_;   // the same of the only head, where its parts may leave one by one
  std::vector<HeadOut> heads_;
  std::vector<void*> allocs_;
  std::vector<void*> pinned_;
  std::vector<std::unique_ptr<cvmk_conv_plan, void (*)(void*)>> plans_;
  std::vector<std::unique_ptr<cvmk_stem_conv_plan, void (*)(void*)>> stem_plans_;
  size_t device_bytes_ = 0;
  // input staging
  void* in_host_ = nullptr;
  void* in_dev_ = nullptr;
  size_t in_bytes_ = 0;
  int32_t* status_dev_ = nullptr;
  int32_t* status_host_ = nullptr;
  GraphExec kernels_exec_;
  bool use_graph_ = true;
  // upload / compute overlap: the copy stream and one event per part of the batch
  cudaStream_t copy_stream_ = nullptr;
  std::vector<cudaEvent_t> part_events_;
  cudaStream_t down_stream_ = nullptr;   // the parts of a head, each behind its part_done_ event
  std::vector<cudaEvent_t> part_done_;
  int32_t* done_host_ = nullptr;    // pinned: the last kernel of an inference has delivered the heads
  void AwaitDone();
  void RunOnce(const void* input, char* out);
  void Settle();
  std::chrono::steady_clock::time_point last_call_;   // the end of the last inference
  std::unique_ptr<HostPool> pool_;   // created by the first inference that has enough bytes to move
  HostPool& pool();
  // How the heads reach the host: small ones are written into page-locked memory by a kernel
  // together with the status word, one large head that goes out as it is by the copy engine in
  // pieces that host threads move on while the next ones arrive, anything else by one copy each.
  enum class Download { kKernel, kPieces, kCopies };
  Download download_ = Download::kCopies;
  bool plain_ = false;
  std::vector<cudaEvent_t> piece_events_;
  size_t download_piece_ = 0;
  std::vector<size_t> piece_end_;   // head bytes up to each piece's end
  size_t queued_pieces_ = 0, arrived_pieces_ = 0, deliver_units_ = 0;   // of the inference that runs
  size_t DeliverUnit() const { return std::min(kStagePiece, download_piece_) / 2; }
  int32_t* valid_host_ = nullptr;    // pinned copy of HeadOut::valid_count
  void ChooseDownload();
  void StartFill(char* out);
  void StartDelivery(char* out);
  void QueuePieces(char* head, size_t bytes, cudaStream_t s);
  void PollPieces();
  void DeliverPieces();
  void DeliverHead(char* out, HostPool* awake);

  void* dalloc(size_t bytes);
  // Activation memory.  Every activation buffer gets a virtual address range of its own when the
  // graph is lowered (kernel descriptors and tensor maps are built on those addresses); once the
  // schedule is known, buffers whose lifetimes do not overlap are backed by the SAME physical
  // memory (CUDA virtual memory management: one physical allocation mapped at several addresses),
  // which is what the reference's storage planner does with its shared pool
  // (src/runtime/graph_runtime.cc:503-610).  Falls back to one cudaMalloc per buffer when the
  // driver's virtual memory calls are not available.
  struct ActBuf {
    void* va = nullptr;
    size_t bytes = 0, va_size = 0;
    uint32_t root = UINT32_MAX;   // node whose lowering made the allocation
    int first = 0, last = 0;      // schedule positions of the first write and the last read
    int first0 = 0, last0 = 0;    // the same before the chunked prefix stretched them
    size_t mapped = 0;            // bytes of it that have physical memory
  };
  struct PhysBlock { unsigned long long handle = 0; size_t size = 0; int free_at = 0; };
  void* dalloc_activation(size_t bytes, uint32_t root);
  void MapActivations();
  void UnmapActivations();
  // Lifetimes for a chunked prefix of `prefix` steps (everything those steps touch lives across
  // all of them), then the physical backing; whatever was mapped before is released first.
  void PlanForPrefix(size_t prefix);
  std::vector<int> step_pos_;   // step -> schedule position
  std::vector<ActBuf> act_;
  std::vector<PhysBlock> phys_;
  bool vmm_ = false;
  size_t vmm_gran_ = 0;
  // Uploads: BeginUpload() starts the staging of a pageable input (the whole of it), SendRange()
  // queues the transfer of a part, Upload() does both for all of it.
  Source SourceOf(const void* input) const;
  void BeginUpload(const void* input, Source src);
  void SendRange(const void* input, Source src, size_t begin, size_t bytes, cudaStream_t s);
  void Upload(const void* input, cudaStream_t s);
  void Enqueue(cudaStream_t s, size_t first = 0);
  friend struct Lowering;
};

}  // namespace cvm
