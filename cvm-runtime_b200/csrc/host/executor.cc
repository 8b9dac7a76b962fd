// Lowering of a Graph into kernel launches, and the per-inference replay.
#include "executor.h"
#include <cuda.h>
#include <algorithm>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <map>
#include <thread>

namespace cvm {

#define CUDA_OK(expr)                                                                      \
  do {                                                                                     \
    cudaError_t e__ = (expr);                                                              \
    CHECK(e__ == cudaSuccess) << "CUDA: " << #expr << ": " << cudaGetErrorString(e__);     \
  } while (0)

#define KERNEL_OK(expr)                                                                    \
  do {                                                                                     \
    int rc__ = (expr);                                                                     \
    CHECK(rc__ == CVMK_OK) << "kernel launcher failed (" << rc__ << "): " << cvmk_last_error(); \
  } while (0)

namespace {

bool nhwc_equiv(const Shape& s) {  // NCHW and NHWC orders coincide
  return s.size() == 4 && ((s[2] == 1 && s[3] == 1) || s[1] == 1);
}
bool wants_nhwc(const Shape& s) { return s.size() == 4 && !nhwc_equiv(s); }

// Element stride of every logical dimension in the buffer's physical layout.
std::vector<int64_t> phys_strides(const Shape& s, bool nhwc) {
  std::vector<int64_t> st(s.size(), 1);
  if (nhwc) {
    st[1] = 1;
    st[3] = s[1];
    st[2] = s[3] * s[1];
    st[0] = s[2] * s[3] * s[1];
  } else {
    for (int i = (int)s.size() - 2; i >= 0; --i) st[i] = st[i + 1] * s[i + 1];
  }
  return st;
}
// Logical dimensions in physical order, outermost first.
std::vector<int> phys_order(const Shape& s, bool nhwc) {
  std::vector<int> o(s.size());
  for (size_t i = 0; i < s.size(); ++i) o[i] = (int)i;
  if (nhwc) o = {0, 2, 3, 1};
  return o;
}

void plan_deleter(void* p) { free(p); }

}  // namespace

void* Executor::dalloc(size_t bytes) {
  void* p = nullptr;
  const size_t sz = std::max<size_t>((bytes + 255) / 256 * 256, 256);
  CUDA_OK(cudaMalloc(&p, sz));
  allocs_.push_back(p);
  device_bytes_ += sz;
  return p;
}

// ---- CUDA virtual memory management, through the driver entry points -------------------------
namespace {
struct Vmm {
  CUresult (*get_granularity)(size_t*, const CUmemAllocationProp*, CUmemAllocationGranularity_flags) = nullptr;
  CUresult (*reserve)(CUdeviceptr*, size_t, size_t, CUdeviceptr, unsigned long long) = nullptr;
  CUresult (*address_free)(CUdeviceptr, size_t) = nullptr;
  CUresult (*create)(CUmemGenericAllocationHandle*, size_t, const CUmemAllocationProp*, unsigned long long) = nullptr;
  CUresult (*release)(CUmemGenericAllocationHandle) = nullptr;
  CUresult (*map)(CUdeviceptr, size_t, size_t, CUmemGenericAllocationHandle, unsigned long long) = nullptr;
  CUresult (*unmap)(CUdeviceptr, size_t) = nullptr;
  CUresult (*set_access)(CUdeviceptr, size_t, const CUmemAccessDesc*, size_t) = nullptr;
  bool ok = false;
};
const Vmm& vmm() {
  static Vmm v = [] {
    Vmm t;
    auto get = [](const char* name) {
      void* fn = nullptr;
      cudaDriverEntryPointQueryResult q;
      if (cudaGetDriverEntryPoint(name, &fn, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) fn = nullptr;
      return fn;
    };
    t.get_granularity = reinterpret_cast<decltype(t.get_granularity)>(get("cuMemGetAllocationGranularity"));
    t.reserve = reinterpret_cast<decltype(t.reserve)>(get("cuMemAddressReserve"));
    t.address_free = reinterpret_cast<decltype(t.address_free)>(get("cuMemAddressFree"));
    t.create = reinterpret_cast<decltype(t.create)>(get("cuMemCreate"));
    t.release = reinterpret_cast<decltype(t.release)>(get("cuMemRelease"));
    t.map = reinterpret_cast<decltype(t.map)>(get("cuMemMap"));
    t.unmap = reinterpret_cast<decltype(t.unmap)>(get("cuMemUnmap"));
    t.set_access = reinterpret_cast<decltype(t.set_access)>(get("cuMemSetAccess"));
    t.ok = t.get_granularity && t.reserve && t.address_free && t.create && t.release && t.map && t.unmap && t.set_access;
    cudaGetLastError();
    return t;
  }();
  return v;
}
CUmemAllocationProp device_prop(int device) {
  CUmemAllocationProp prop;
  memset(&prop, 0, sizeof(prop));
  prop.type = CU_MEM_ALLOCATION_TYPE_PINNED;
  prop.location.type = CU_MEM_LOCATION_TYPE_DEVICE;
  prop.location.id = device;
  return prop;
}
}  // namespace

void* Executor::dalloc_activation(size_t bytes, uint32_t root) {
  // small buffers are not worth a mapping of their own (the granularity is 2 MiB)
  if (!vmm_ || bytes < (size_t)1 << 20) return dalloc(bytes);
  ActBuf a;
  a.bytes = std::max<size_t>(bytes, 256);
  a.va_size = (a.bytes + vmm_gran_ - 1) / vmm_gran_ * vmm_gran_;
  a.root = root;
  CUdeviceptr va = 0;
  const CUresult r = vmm().reserve(&va, a.va_size, vmm_gran_, 0, 0);
  CHECK(r == CUDA_SUCCESS) << "cuMemAddressReserve(" << a.va_size << ") failed (" << (int)r << ")";
  a.va = reinterpret_cast<void*>(va);
  act_.push_back(a);
  return a.va;
}

// Backs the activation buffers with physical memory in chunks of the allocation granularity (2 MiB):
// walking the buffers in the order of their first write, a buffer takes any chunks that are free by
// then (most recently freed first: they are the likeliest to be still in L2) and new ones for the
// rest; its chunks are free again after its last read.  Chunks need not be contiguous -- the
// virtual range of a buffer is -- so nothing is lost to fragmentation.
void Executor::PlanForPrefix(size_t prefix) {
  if (!vmm_ || act_.empty()) return;
  UnmapActivations();
  const int p = prefix > 0 ? step_pos_[std::min(prefix, step_pos_.size()) - 1] : -2;   // (heads' steps have no position)
  for (auto& a : act_) {
    a.first = a.first0;
    a.last = a.last0;
    if (a.first <= p) { a.first = -1; a.last = std::max(a.last, p); }
  }
  MapActivations();
}

void Executor::UnmapActivations() {
  for (auto& a : act_) {
    if (a.mapped) vmm().unmap(reinterpret_cast<CUdeviceptr>(a.va), a.mapped);
    a.mapped = 0;
  }
  for (auto& b : phys_) {
    vmm().release((CUmemGenericAllocationHandle)b.handle);
    device_bytes_ -= b.size;
  }
  phys_.clear();
}

void Executor::MapActivations() {
  if (!vmm_ || act_.empty()) return;
  const CUmemAllocationProp prop = device_prop(device_);
  CUmemAccessDesc access;
  memset(&access, 0, sizeof(access));
  access.location = prop.location;
  access.flags = CU_MEM_ACCESS_FLAGS_PROT_READWRITE;
  std::vector<size_t> order(act_.size());
  for (size_t i = 0; i < order.size(); ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](size_t x, size_t y) { return act_[x].first < act_[y].first; });
  for (size_t i : order) {
    ActBuf& a = act_[i];
    const size_t need = a.va_size / vmm_gran_;
    std::vector<int> cand;
    for (size_t c = 0; c < phys_.size(); ++c)
      if (phys_[c].free_at <= a.first) cand.push_back((int)c);
    std::stable_sort(cand.begin(), cand.end(), [&](int x, int y) { return phys_[x].free_at > phys_[y].free_at; });
    std::vector<int> mine(cand.begin(), cand.begin() + std::min(cand.size(), need));
    while (mine.size() < need) {
      PhysBlock nb;
      CUmemGenericAllocationHandle h = 0;
      const CUresult r = vmm().create(&h, vmm_gran_, &prop, 0);
      CHECK(r == CUDA_SUCCESS) << "cuMemCreate failed (" << (int)r << ") after " << device_bytes_ << " bytes";
      nb.handle = (unsigned long long)h;
      nb.size = vmm_gran_;
      phys_.push_back(nb);
      device_bytes_ += vmm_gran_;
      mine.push_back((int)phys_.size() - 1);
    }
    const CUdeviceptr va = reinterpret_cast<CUdeviceptr>(a.va);
    for (size_t k = 0; k < need; ++k) {
      phys_[mine[k]].free_at = a.last + 1;
      const CUresult r = vmm().map(va + k * vmm_gran_, vmm_gran_, 0, (CUmemGenericAllocationHandle)phys_[mine[k]].handle, 0);
      CHECK(r == CUDA_SUCCESS) << "cuMemMap failed (" << (int)r << ")";
      a.mapped += vmm_gran_;
    }
    const CUresult r = vmm().set_access(va, a.va_size, &access, 1);
    CHECK(r == CUDA_SUCCESS) << "cuMemSetAccess failed (" << (int)r << ")";
  }
}

// How a batch may be cut for upload / compute overlap: five parts (an eighth, three quarters, an eighth), four
// (1/8, 1/4, 5/16, 5/16) or two (3/8, 5/8), as indices into Lowering::batch_ranges().  Where the kernels take
// longer than the upload, what counts is how soon the first part is there and how few launches each step takes;
// where the upload takes longer, how little is left to do when the last part has arrived.  Measured at load
// (ChooseSchedules); against five parts always: ResNet-50, 256 images 2389 -> 2321 us (four parts), VGG-19, 32
// images 865 -> 835 (two).
const std::vector<int> kCuts[] = {{0, 1, 2, 3, 4}, {0, 1, 5, 6}, {7, 8}};
constexpr size_t kMaxParts = 5;

struct Lowering {
  Executor& ex;
  const Graph& g;
  std::vector<DevBuf> buf;
  std::vector<int> uses;
  std::vector<char> is_head, safe8, absorbed;
  uint32_t data_eid = 0;
  uint32_t cur_root = UINT32_MAX;   // node being lowered: tags the activation buffers it allocates
  std::vector<uint32_t> root_of;    // node -> root of the fused group it runs in
  // activation memory: planned when a node is being lowered, persistent otherwise (heads, staging)
  void* act_alloc(size_t bytes) { return cur_root == UINT32_MAX ? ex.dalloc(bytes) : ex.dalloc_activation(bytes, cur_root); }
  DevBuf raw_in;          // the input exactly as the C-ABI delivers it (row-major int8 / int32)
  int32_t data_range = 127;

  Lowering(Executor& e, const Graph& gr) : ex(e), g(gr) {}

  // The parts of the batch that steps are prepared for, as ranges of images in the order of kCuts (none for
  // batches under eight images).
  struct Range { int64_t begin, end; };
  static std::vector<Range> batch_ranges(int64_t n) {
    if (n < 8 || dev_env("CVM_B200_NO_UPLOAD_OVERLAP")) return {};
    const int at[][2] = {{0, 2}, {2, 6}, {6, 10}, {10, 14}, {14, 16}, {6, 11}, {11, 16}, {0, 6}, {6, 16}};   // sixteenths
    std::vector<Range> r;
    for (const auto& a : at) r.push_back({(n * a[0] + 8) / 16, (n * a[1] + 8) / 16});
    return r;
  }
  void input_ranges(const std::vector<Range>& parts, size_t image_bytes) {
    if (parts.empty()) return;
    ex.range_end_.clear();
    for (const Range& r : parts) ex.range_end_.push_back((size_t)r.end * image_bytes);
  }

  void add_step(const std::string& label, std::function<int(cudaStream_t)> fn) {
    ex.steps_.push_back({label, std::move(fn), {}});
  }
  // The launch of a convolution on one part of the batch.  Its plan (tensor maps and more) is prepared when a
  // schedule first captures the part: most steps of a network are never run in parts.
  template <typename Plan, typename Desc>
  static std::function<int(cudaStream_t)> part_launch(const Desc& desc, int (*prepare)(const Desc*, Plan*),
                                                      int (*launch)(const Plan*, cvmk_stream_t)) {
    std::shared_ptr<Plan> plan;
    return [=](cudaStream_t s) mutable {
      if (!plan) {
        void* mem = nullptr;
        CHECK(posix_memalign(&mem, 64, sizeof(Plan)) == 0);
        plan.reset((Plan*)mem, plan_deleter);
        const int rc = prepare(&desc, plan.get());
        if (rc != CVMK_OK) {
          plan.reset();
          return rc;
        }
      }
      return launch(plan.get(), s);
    };
  }
  // ------------------------------------------------------------------ analysis
  void analyse() {
    const uint32_t ne = g.num_entries;
    buf.assign(ne, DevBuf());
    uses.assign(ne, 0);
    is_head.assign(ne, 0);
    safe8.assign(ne, 0);
    absorbed.assign(g.nodes.size(), 0);
    for (const auto& n : g.nodes)
      for (const auto& e : n.inputs) uses[g.entry_id(e)]++;
    for (const auto& e : g.outputs) is_head[g.entry_id(e)] = 1;
    for (uint32_t nid = 0; nid < g.nodes.size(); ++nid) {
      const Node& n = g.nodes[nid];
      const uint32_t e0 = g.entry_id(nid, 0);
      auto in_safe = [&](size_t i) { return (bool)safe8[g.entry_id(n.inputs[i])]; };
      if (n.is_variable()) { safe8[e0] = g.precision[e0] <= 8; continue; }
      const std::string& op = n.op->name;
      bool s = false;
      if (op == "cvm_clip" || op == "cvm_left_shift") s = n.attrs.i("precision") <= 8;
      else if (op == "clip") s = n.attrs.i("a_min") >= -127 && n.attrs.i("a_max") <= 127;
      else if (op == "cvm_right_shift") {
        const int64_t p = n.attrs.i("precision"), b = n.attrs.i("shift_bit");
        s = p == 1 || b >= 31 || (p <= 8 && p + b < 32);
      } else if (op == "relu" || op == "max_pool2d" || op == "upsampling" || op == "flatten" ||
                 op == "reshape" || op == "squeeze" || op == "expand_dims" || op == "abs" ||
                 op == "negative" || op == "max") s = in_safe(0);
      else if (op == "concatenate" || op == "broadcast_max") {
        s = true;
        for (size_t i = 0; i < n.inputs.size(); ++i) s = s && in_safe(i);
      } else if (op == "transpose" || op == "strided_slice" || op == "slice_like" || op == "repeat" ||
                 op == "tile" || op == "take") s = in_safe(0);
      else if (op == "cvm_lut") s = in_safe(1);
      else if (op == "where") s = in_safe(1) && in_safe(2);
      else if (op == "cvm_precision" || op == "broadcast_greater") s = true;
      safe8[e0] = s;
    }
    for (uint32_t e = 0; e < ne; ++e) {
      buf[e].shape = g.shape[e];
      buf[e].dtype = safe8[e] ? CVMK_I8 : CVMK_I32;
      buf[e].nhwc = wants_nhwc(g.shape[e]);
    }
    // transpose(0, 2, 3, 1) of a tensor stored channels-last: the row-major bytes of the result ARE
    // the input's bytes.  The result is therefore kept row-major (not channels-last again, which
    // would shuffle it once here and once more at the reshape that usually follows: the detection
    // heads of SSD do this twelve times per step) and the node becomes an alias.
    for (uint32_t nid = 0; nid < g.nodes.size(); ++nid)
      if (transpose_is_identity(nid)) buf[g.entry_id(nid, 0)].nhwc = false;
  }

  // true for transpose nodes with axes (0, 2, 3, 1) over a 4-D input that is stored channels-last
  bool transpose_is_identity(uint32_t nid) {
    const Node& n = g.nodes[nid];
    if (n.is_variable() || n.op->name != "transpose" || n.inputs.size() != 1) return false;
    const uint32_t ei = g.entry_id(n.inputs[0]);
    if (g.shape[ei].size() != 4 || !buf[ei].nhwc || g.params.count(ei)) return false;
    const Shape axes = n.attrs.t("axes");
    if (!(axes.size() == 4 && axes[0] == 0 && axes[1] == 2 && axes[2] == 3 && axes[3] == 1)) return false;
    // only when every reader takes the tensor by its layout flag: the reshape-like operators (and
    // the output copy of a graph head); convolutions and pooling expect channels-last operands
    const uint32_t eo = g.entry_id(nid, 0);
    for (uint32_t m = nid + 1; m < g.nodes.size(); ++m) {
      const Node& c = g.nodes[m];
      if (c.is_variable()) continue;
      for (const auto& e : c.inputs) {
        if (g.entry_id(e) != eo) continue;
        const std::string& op = c.op->name;
        if (op != "flatten" && op != "reshape" && op != "squeeze" && op != "expand_dims") return false;
      }
    }
    return true;
  }

  // ------------------------------------------------------------------ buffers
  DevBuf& materialize(uint32_t eid) {
    DevBuf& b = buf[eid];
    if (b.ptr) return b;
    auto it = g.params.find(eid);
    b.ptr = it != g.params.end() ? ex.dalloc(b.bytes()) : act_alloc(b.bytes());
    if (it != g.params.end()) {
      // parameter: convert on the host into the entry's dtype and layout, upload once
      const HostTensor& t = it->second;
      const int64_t n = shape_size(b.shape);
      std::vector<int32_t> phys(n);
      if (b.nhwc) {
        const int64_t C = b.shape[1], H = b.shape[2], W = b.shape[3];
        for (int64_t i = 0; i < n; ++i) {
          const int64_t w = i % W, h = (i / W) % H, c = (i / (W * H)) % C, nn = i / (W * H * C);
          phys[((nn * H + h) * W + w) * C + c] = t.data[i];
        }
      } else {
        phys = t.data;
      }
      if (b.dtype == CVMK_I8) {
        std::vector<int8_t> p8(n);
        for (int64_t i = 0; i < n; ++i) p8[i] = (int8_t)phys[i];
        CUDA_OK(cudaMemcpy(b.ptr, p8.data(), n, cudaMemcpyHostToDevice));
      } else {
        CUDA_OK(cudaMemcpy(b.ptr, phys.data(), n * 4, cudaMemcpyHostToDevice));
      }
    }
    return b;
  }

  // Same logical tensor copied between two buffers that may differ in layout and dtype.
  void emit_convert(const DevBuf& src, const DevBuf& dst, const std::string& label,
                    const cvmk_epilogue* ep = nullptr) {
    if (src.nhwc == dst.nhwc && src.shape == dst.shape) {
      // same element order on both sides: the vectorised contiguous kernel does it
      cvmk_epilogue e;
      memset(&e, 0, sizeof(e));
      if (ep) e = *ep;
      const DevBuf a = src, b = dst;
      const int64_t cnt = shape_size(dst.shape);
      add_step(label, [a, b, e, cnt](cudaStream_t s_) {
        return cvmk_elemwise(a.ptr, a.dtype, b.ptr, b.dtype, cnt, &e, s_);
      });
      return;
    }
    // NCHW <-> NHWC of one element type: a batched matrix transpose through shared memory
    if (src.nhwc != dst.nhwc && src.shape == dst.shape && src.shape.size() == 4 && src.dtype == dst.dtype &&
        (!ep || ep->n == 0 || (ep->n == 1 && ep->s[0].op == CVMK_EP_CLIP)) && !dev_env("CVM_B200_NO_TILED_TRANSPOSE")) {
      const Shape& sh = src.shape;
      const int64_t batch = sh[0];
      const int64_t c = sh[1], hw = sh[2] * sh[3];
      const int rows = (int)(src.nhwc ? hw : c), cols = (int)(src.nhwc ? c : hw);
      const int clamp = ep && ep->n == 1;
      const int lo = clamp ? ep->s[0].a : 0, hi = clamp ? ep->s[0].b : 0;
      const int dtype = src.dtype;
      const size_t image = (size_t)c * hw * dtype;
      const char* from = (const char*)src.ptr;
      char* to = (char*)dst.ptr;
      auto range = [=](int64_t b0, int64_t b1) {
        return [=](cudaStream_t s_) {
          return cvmk_transpose_batched(from + b0 * image, to + b0 * image, dtype, b1 - b0, rows, cols, clamp, lo, hi, s_);
        };
      };
      add_step(label, range(0, batch));
      if (image % 16 == 0)
        for (const Range& r : batch_ranges(batch)) ex.steps_.back().chunk.push_back(range(r.begin, r.end));
      ex.steps_.back().images = batch;
      return;
    }
    cvmk_strided_desc d;
    memset(&d, 0, sizeof(d));
    d.op = CVMK_OP_COPY;
    const Shape& s = dst.shape;
    const auto order = phys_order(s, dst.nhwc);
    const auto ss = phys_strides(src.shape, src.nhwc), ds = phys_strides(s, dst.nhwc);
    d.ndim = (int)s.size();
    for (int k = 0; k < d.ndim; ++k) {
      d.extent[k] = s[order[k]];
      d.a_stride[k] = ss[order[k]];
      d.y_stride[k] = ds[order[k]];
    }
    d.a = src.ptr; d.a_dtype = src.dtype;
    d.y = dst.ptr; d.y_dtype = dst.dtype;
    if (ep) d.ep = *ep;
    add_step(label, [d](cudaStream_t s_) { return cvmk_strided(&d, s_); });
  }

  // A row-major view of an entry; converts into a temporary when the entry is channels-last.
  DevBuf canon_view(uint32_t eid, const std::string& label) {
    DevBuf& b = materialize(eid);
    if (!b.nhwc) return b;
    DevBuf t = b;
    t.nhwc = false;
    t.ptr = act_alloc(t.bytes());
    emit_convert(b, t, label + ":to_rowmajor");
    return t;
  }
  // int32 row-major view (get_valid_counts / nms operands).
  DevBuf canon_i32_view(uint32_t eid, const std::string& label) {
    DevBuf& b = materialize(eid);
    if (!b.nhwc && b.dtype == CVMK_I32) return b;
    DevBuf t = b;
    t.nhwc = false;
    t.dtype = CVMK_I32;
    t.ptr = act_alloc(t.bytes());
    emit_convert(b, t, label + ":to_i32");
    return t;
  }
  // int8 view in the entry's own layout; narrows like static_cast<int8_t> when stored as int32.
  DevBuf i8_view(uint32_t eid, const std::string& label) {
    DevBuf& b = materialize(eid);
    if (b.dtype == CVMK_I8) return b;
    DevBuf t = b;
    t.dtype = CVMK_I8;
    t.ptr = act_alloc(t.bytes());
    const DevBuf src = b;
    const int64_t n = shape_size(b.shape);
    add_step(label + ":narrow", [src, t, n](cudaStream_t s) {
      return cvmk_elemwise(src.ptr, src.dtype, t.ptr, t.dtype, n, nullptr, s);
    });
    return t;
  }

  // ------------------------------------------------------------------ chains
  struct Chain {
    cvmk_epilogue ep;
    uint32_t tail_eid;
    uint32_t tail_nid;
  };

  bool scalar_param(uint32_t eid, int32_t* v) const {
    auto it = g.params.find(eid);
    if (it == g.params.end() || it->second.data.size() != 1) return false;
    *v = it->second.data[0];
    return true;
  }

  // Translate node `nid`, consuming entry `cur`, into one chain step.  False if not expressible.
  bool node_as_step(uint32_t nid, uint32_t cur, cvmk_ep_step* st) {
    const Node& n = g.nodes[nid];
    const std::string& op = n.op->name;
    memset(st, 0, sizeof(*st));
    auto alpha = [&](int64_t p) { return (int32_t)((((int64_t)1) << (p - 1)) - 1); };
    if (op == "relu") st->op = CVMK_EP_RELU;
    else if (op == "abs") st->op = CVMK_EP_ABS;
    else if (op == "negative") st->op = CVMK_EP_NEG;
    else if (op == "cvm_precision") st->op = CVMK_EP_PRECISION;
    else if (op == "clip") { st->op = CVMK_EP_CLIP; st->a = (int32_t)n.attrs.i("a_min"); st->b = (int32_t)n.attrs.i("a_max"); }
    else if (op == "cvm_clip") { st->op = CVMK_EP_CLIP; st->b = alpha(n.attrs.i("precision")); st->a = -st->b; }
    else if (op == "cvm_right_shift") { st->op = CVMK_EP_RSHIFT; st->a = (int32_t)n.attrs.i("shift_bit"); st->b = (int32_t)n.attrs.i("precision"); }
    else if (op == "cvm_left_shift") { st->op = CVMK_EP_LSHIFT; st->a = (int32_t)n.attrs.i("shift_bit"); st->b = (int32_t)n.attrs.i("precision"); }
    else if (op == "elemwise_add" || op == "elemwise_sub") {
      const uint32_t e0 = g.entry_id(n.inputs[0]), e1 = g.entry_id(n.inputs[1]);
      if (e0 == e1) return false;
      const uint32_t other = e0 == cur ? e1 : e0;
      if (op == "elemwise_add") st->op = CVMK_EP_ADD_T;
      else st->op = e0 == cur ? CVMK_EP_SUB_T : CVMK_EP_RSUB_T;
      st->ptr = reinterpret_cast<const void*>((uintptr_t)other + 1);  // resolved in bind_chain()
    } else if (op.compare(0, 10, "broadcast_") == 0) {
      const uint32_t e0 = g.entry_id(n.inputs[0]), e1 = g.entry_id(n.inputs[1]);
      if (e0 == e1) return false;
      const uint32_t other = e0 == cur ? e1 : e0;
      int32_t v;
      if (!scalar_param(other, &v)) return false;
      if (g.shape[g.entry_id(nid, 0)] != g.shape[cur]) return false;
      const bool lhs = e0 == cur;
      if (op == "broadcast_add") { st->op = CVMK_EP_ADD_S; st->a = v; }
      else if (op == "broadcast_sub") {
        if (lhs) { st->op = CVMK_EP_ADD_S; st->a = (int32_t)(0u - (uint32_t)v); }
        else { st->op = CVMK_EP_RSUB_S; st->a = v; }
      } else if (op == "broadcast_mul") { st->op = CVMK_EP_MUL_S; st->a = v; }
      else if (op == "broadcast_max") { st->op = CVMK_EP_MAX_S; st->a = v; }
      else if (op == "broadcast_div") { st->op = lhs ? CVMK_EP_DIV_S : CVMK_EP_RDIV_S; st->a = v; }
      else if (op == "broadcast_greater") { st->op = lhs ? CVMK_EP_GT_S : CVMK_EP_LT_S; st->a = v; }
      else return false;
    } else {
      return false;
    }
    return true;
  }

  // non_max_suppression nodes that overwrite rows of their INPUT entry (the CPU operator's side
  // effect, nms.cc:93-97, reproduced when that entry is read again): (node, entry) pairs.  They are
  // the only in-place writers of the graph, so they are the only thing a deferred read can miss.
  std::vector<std::pair<uint32_t, uint32_t>> input_writers;
  void find_input_writers() {
    for (uint32_t nid = 0; nid < g.nodes.size(); ++nid) {
      const Node& n = g.nodes[nid];
      if (n.is_variable() || n.op->name != "non_max_suppression" || n.attrs.i("top_k") <= 0) continue;
      const uint32_t in_eid = g.entry_id(n.inputs[0]);
      bool observed = false;
      for (const auto& h : g.outputs) observed |= g.entry_id(h) == in_eid;
      for (uint32_t m = nid + 1; m < g.nodes.size(); ++m)
        for (const auto& e : g.nodes[m].inputs) observed |= g.entry_id(e) == in_eid;
      if (observed) input_writers.emplace_back(nid, in_eid);
    }
  }

  // Greedily absorb single-consumer element-wise successors of entry `start`.  A fused group runs
  // at the position of its last member, so every read of the group happens there: a member that
  // reads an entry BEFORE a node that overwrites it in place must not be carried past that node.
  void extend_chain(Chain* c) {
    std::vector<std::pair<uint32_t, uint32_t>> reads;   // (entry, reading node)
    for (const auto& e : g.nodes[c->tail_nid].inputs) reads.emplace_back(g.entry_id(e), c->tail_nid);
    while (c->ep.n < CVMK_MAX_EP_STEPS) {
      const uint32_t cur = c->tail_eid;
      if (is_head[cur] || uses[cur] != 1) break;
      uint32_t consumer = UINT32_MAX;
      for (uint32_t nid = c->tail_nid + 1; nid < g.nodes.size() && consumer == UINT32_MAX; ++nid)
        for (const auto& e : g.nodes[nid].inputs)
          if (g.entry_id(e) == cur) { consumer = nid; break; }
      if (consumer == UINT32_MAX || absorbed[consumer]) break;  // e.g. a join taken by its other branch
      bool crosses_writer = false;
      for (const auto& w : input_writers)
        for (const auto& r : reads)
          crosses_writer |= r.first == w.second && r.second < w.first && w.first < consumer;
      if (crosses_writer) break;
      cvmk_ep_step st;
      if (!node_as_step(consumer, cur, &st)) break;
      for (const auto& e : g.nodes[consumer].inputs)
        if (g.entry_id(e) != cur) reads.emplace_back(g.entry_id(e), consumer);
      c->ep.s[c->ep.n++] = st;
      absorbed[consumer] = 1;
      c->tail_nid = consumer;
      c->tail_eid = g.entry_id(consumer, 0);
    }
  }

  // Replace the entry placeholders of *_T steps by device pointers.
  void bind_chain(cvmk_epilogue* ep) {
    for (int i = 0; i < ep->n; ++i) {
      cvmk_ep_step& s = ep->s[i];
      if (s.op == CVMK_EP_ADD_T || s.op == CVMK_EP_SUB_T || s.op == CVMK_EP_RSUB_T) {
        const uint32_t other = (uint32_t)((uintptr_t)s.ptr - 1);
        DevBuf& o = materialize(other);
        s.ptr = o.ptr;
        s.ptr_dtype = o.dtype;
      }
    }
  }

  // ------------------------------------------------------------------ operators
  const int32_t* bias_vector(uint32_t eid) {
    auto it = g.params.find(eid);
    if (it != g.params.end()) {  // the usual case: upload the int32 vector once
      const auto& v = it->second.data;
      // zero padded to a multiple of 32 entries: a convolution whose output channels are padded
      // for the tensor-core kernel reads that far
      const size_t padded = (v.size() + 31) / 32 * 32;
      void* p = ex.dalloc(padded * 4);
      CUDA_OK(cudaMemset(p, 0, padded * 4));
      CUDA_OK(cudaMemcpy(p, v.data(), v.size() * 4, cudaMemcpyHostToDevice));
      return reinterpret_cast<const int32_t*>(p);
    }
    DevBuf b = canon_i32_view(eid, "bias");
    return reinterpret_cast<const int32_t*>(b.ptr);
  }

  void lower_conv_like(uint32_t nid, bool dense) {
    const Node& n = g.nodes[nid];
    const uint32_t ex_ = g.entry_id(n.inputs[0]), ew = g.entry_id(n.inputs[1]);
    const bool use_bias = n.attrs.b("use_bias");
    const Shape& xs = g.shape[ex_];
    const Shape& wsh = g.shape[ew];
    auto wit = g.params.find(ew);
    CHECK(wit != g.params.end()) << n.op->name << " " << n.name() << ": weights must be a parameter";
    const HostTensor& wt = wit->second;

    int N, H, W, C, OC, KH, KW, OH, OW, groups, sh, sw, ph, pw, dh, dw;
    if (dense) {
      N = (int)xs[0]; H = W = 1; C = (int)xs[1]; OC = (int)wsh[0]; KH = KW = 1; OH = OW = 1; groups = 1;
      sh = sw = dh = dw = 1; ph = pw = 0;
    } else {
      const Shape& os = g.shape[g.entry_id(nid, 0)];
      N = (int)xs[0]; C = (int)xs[1]; H = (int)xs[2]; W = (int)xs[3];
      OC = (int)wsh[0]; KH = (int)wsh[2]; KW = (int)wsh[3]; OH = (int)os[2]; OW = (int)os[3];
      groups = (int)n.attrs.i("groups");
      sh = (int)n.attrs.t("strides")[0]; sw = (int)n.attrs.t("strides")[1];
      ph = (int)n.attrs.t("padding")[0]; pw = (int)n.attrs.t("padding")[1];
      dh = (int)n.attrs.t("dilation")[0]; dw = (int)n.attrs.t("dilation")[1];
    }
    const int icg = C / groups;

    Chain ch;
    memset(&ch.ep, 0, sizeof(ch.ep));
    ch.tail_eid = g.entry_id(nid, 0);
    ch.tail_nid = nid;
    if (use_bias) {
      ch.ep.s[0].op = CVMK_EP_ADD_C;
      ch.ep.s[0].ptr = bias_vector(g.entry_id(n.inputs[2]));
      ch.ep.n = 1;
    }
    extend_chain(&ch);
    bind_chain(&ch.ep);
    DevBuf& out = materialize(ch.tail_eid);
    const std::string label = n.op->name + ":" + n.name();

    cvmk_conv_desc probe;
    memset(&probe, 0, sizeof(probe));
    probe.N = N; probe.H = H; probe.W = W; probe.C = C; probe.OC = OC; probe.KH = KH; probe.KW = KW;
    probe.OH = OH; probe.OW = OW; probe.stride_h = sh; probe.stride_w = sw; probe.pad_h = ph; probe.pad_w = pw;
    probe.dil_h = dh; probe.dil_w = dw;
    // |sum + bias| can never exceed this: int8 operands (|x| <= 128 even after a narrowing view)
    // and the bias values themselves when they are parameters.
    {
      int64_t bias_max = 0;
      if (use_bias) {
        const uint32_t eb = g.entry_id(n.inputs[2]);
        auto bit = g.params.find(eb);
        if (bit != g.params.end()) {
          for (int32_t v : bit->second.data) bias_max = std::max<int64_t>(bias_max, std::llabs((long long)v));
        } else {
          bias_max = ((int64_t)1 << (g.precision[eb] - 1)) - 1;
        }
      }
      probe.acc_bound = (int64_t)icg * KH * KW * 128 * 128 + bias_max;
      probe.bias_static = (!use_bias || g.params.count(g.entry_id(n.inputs[2])) > 0) ? 1 : 0;
    }
    const bool depthwise = !dense && groups == C && OC == C && C % 16 == 0 && safe8[ex_];
    const bool tc = groups == 1 && cvmk_conv2d_tc_supported(&probe) && !dev_env("CVM_B200_NO_TC");
    // Few-channel convolutions (image stems): gather patches into a [M, Kp] matrix, then run the
    // tensor-core kernel on it as a 1x1 convolution.
    const int kflat = KH * KW * icg, kp = kflat > 64 ? (kflat + 63) / 64 * 64 : (kflat + 31) / 32 * 32;
    cvmk_conv_desc packed = probe;
    packed.N = N * OH * OW; packed.H = packed.W = 1; packed.C = kp; packed.KH = packed.KW = 1;
    packed.OH = packed.OW = 1; packed.stride_h = packed.stride_w = 1; packed.pad_h = packed.pad_w = 0;
    packed.dil_h = packed.dil_w = 1;
    const bool via_pack = !tc && !dense && groups == 1 && safe8[ex_] && C <= 255 && kflat <= 8192 &&
                          (KW - 1) * dw <= 4095 && (KH - 1) * dh <= 2047 &&
                          cvmk_conv2d_tc_supported(&packed) && !dev_env("CVM_B200_NO_TC");

    // Output channel counts the tensor-core kernel does not take (not a multiple of 8: detection
    // heads with anchors x classes channels) run on it with zero weight rows up to a multiple of
    // 32 and a copy of the real channels afterwards, when nothing in the chain indexes the
    // output tensor (no fused tensor operand) and the bias is a parameter.
    const int OCp = (OC + 31) / 32 * 32;
    bool tc_pad = false;
    if (!tc && !dense && groups == 1 && OC % 8 != 0 && !depthwise && !dev_env("CVM_B200_NO_TC")) {
      cvmk_conv_desc pp = probe;
      pp.OC = OCp;
      bool plain_chain = true;
      for (int i = 0; i < ch.ep.n; ++i)
        plain_chain &= !(ch.ep.s[i].op == CVMK_EP_ADD_T || ch.ep.s[i].op == CVMK_EP_SUB_T || ch.ep.s[i].op == CVMK_EP_RSUB_T);
      const bool bias_param = !use_bias || g.params.count(g.entry_id(n.inputs[2])) > 0;
      tc_pad = cvmk_conv2d_tc_supported(&pp) && plain_chain && bias_param && safe8[ex_] && out.shape.size() == 4;
    }
    // weights: OIHW int32 -> int8, [OC, KH, KW, C/groups] (depthwise: [KH, KW, C])
    std::vector<int8_t> w8((size_t)(tc_pad ? OCp : OC) * KH * KW * icg, 0);
    if (depthwise && !tc) {
      for (int c = 0; c < C; ++c)
        for (int k = 0; k < KH * KW; ++k) w8[(size_t)k * C + c] = (int8_t)wt.data[(size_t)c * KH * KW + k];
    } else {
      for (int o = 0; o < OC; ++o)
        for (int i = 0; i < icg; ++i)
          for (int k = 0; k < KH * KW; ++k)
            w8[((size_t)o * KH * KW + k) * icg + i] = (int8_t)wt.data[((size_t)o * icg + i) * KH * KW + k];
    }
    if (via_pack) {  // rows padded with zeros from K to Kp
      std::vector<int8_t> wp((size_t)OC * kp, 0);
      for (int o = 0; o < OC; ++o) memcpy(&wp[(size_t)o * kp], &w8[(size_t)o * kflat], kflat);
      w8.swap(wp);
    }
    int8_t* wdev = (int8_t*)ex.dalloc(w8.size());
    CUDA_OK(cudaMemcpy(wdev, w8.data(), w8.size(), cudaMemcpyHostToDevice));

    // Stem on the tensor cores without a patch matrix: the network input itself, few channels.
    if (via_pack && ex_ == data_eid && raw_in.dtype == CVMK_I8 && dh == 1 && dw == 1 && out.dtype == CVMK_I8 &&
        !dev_env("CVM_B200_NO_STEM_FUSED")) {
      cvmk_stem_conv_desc sd;
      memset(&sd, 0, sizeof(sd));
      sd.x = (const int8_t*)raw_in.ptr; sd.y = out.ptr;
      sd.N = N; sd.H = H; sd.W = W; sd.C = C; sd.OC = OC; sd.KH = KH; sd.KW = KW; sd.OH = OH; sd.OW = OW;
      sd.stride_h = sh; sd.stride_w = sw; sd.pad_h = ph; sd.pad_w = pw;
      sd.clamp = data_range;
      sd.status = ex.status_dev_;
      sd.acc_bound = probe.acc_bound;
      sd.bias_static = probe.bias_static;
      sd.ep = ch.ep;
      if (W % 16 != 0) sd.x_pitch = (W + 15) / 16 * 16;   // TMA rows start on 16-byte boundaries: the rows are moved apart first
      if (cvmk_conv2d_stem_supported(&sd)) {
        std::vector<int8_t> ws((size_t)cvmk_conv2d_stem_weight_bytes(&sd), 0);
        KERNEL_OK(cvmk_conv2d_stem_pack_weights(&sd, wt.data.data(), ws.data()));
        int8_t* wsdev = (int8_t*)ex.dalloc(ws.size());
        CUDA_OK(cudaMemcpy(wsdev, ws.data(), ws.size(), cudaMemcpyHostToDevice));
        sd.w = wsdev;
        // The batch is cut into parts with a plan each, so that an inference can run the stem on the
        // first images while the later ones are still being uploaded.
        const std::vector<Range> parts = (uses[ex_] == 1 && !is_head[ex_]) ? batch_ranges(N) : std::vector<Range>();
        const size_t image = (size_t)C * H * W;
        int8_t* rows = nullptr;
        const int pitch = sd.x_pitch;
        if (pitch > 0) {
          rows = (int8_t*)act_alloc((size_t)N * C * H * pitch);
          sd.x = rows;
          auto move = [this, rows, pitch, image, C, H, W](int64_t b0, int64_t b1) {
            const char* from = (const char*)raw_in.ptr + (size_t)b0 * image;
            char* to = (char*)rows + (size_t)b0 * C * H * pitch;
            const int64_t n = (b1 - b0) * C * H;
            return [from, to, n, W, pitch](cudaStream_t s) { return cvmk_repitch(from, to, n, W, pitch, s); };
          };
          bool aligned = true;
          for (const Range& r : parts) aligned &= ((size_t)r.begin * image) % 4 == 0;
          add_step(label + "[rows]", move(0, N));
          ex.steps_.back().from_input = true;
          for (const Range& r : parts)
            if (aligned) ex.steps_.back().chunk.push_back(move(r.begin, r.end));
          ex.steps_.back().images = N;
        }
        cvmk_stem_conv_plan* plan = nullptr;
        {
          void* mem = nullptr;
          CHECK(posix_memalign(&mem, 64, sizeof(cvmk_stem_conv_plan)) == 0);
          ex.stem_plans_.emplace_back((cvmk_stem_conv_plan*)mem, plan_deleter);
          plan = ex.stem_plans_.back().get();
          KERNEL_OK(cvmk_conv2d_stem_prepare(&sd, plan));
        }
        add_step(label + "[stem]", [plan](cudaStream_t s) { return cvmk_conv2d_stem_launch(plan, s); });
        ex.steps_.back().from_input = pitch == 0;
        ex.steps_.back().images = N;
        for (const Range& r : parts) {   // (whole rows of 16 bytes)
          cvmk_stem_conv_desc cd = sd;
          cd.N = (int)(r.end - r.begin);
          cd.x = sd.x + (size_t)r.begin * C * H * (pitch > 0 ? pitch : W);
          cd.y = (int8_t*)sd.y + (size_t)r.begin * OH * OW * OC;
          ex.steps_.back().chunk.push_back(part_launch(cd, cvmk_conv2d_stem_prepare, cvmk_conv2d_stem_launch));
        }
        input_ranges(parts, image);
        return;
      }
    }

    if (via_pack) {
      int8_t* amat = (int8_t*)act_alloc((size_t)packed.N * kp);
      cvmk_stem_pack_desc sp;
      memset(&sp, 0, sizeof(sp));
      sp.x = (const int8_t*)raw_in.ptr; sp.a = amat;
      sp.N = N; sp.H = H; sp.W = W; sp.C = C; sp.KH = KH; sp.KW = KW; sp.OH = OH; sp.OW = OW;
      sp.stride_h = sh; sp.stride_w = sw; sp.pad_h = ph; sp.pad_w = pw; sp.dil_h = dh; sp.dil_w = dw;
      sp.Kp = kp; sp.clamp = data_range;
      const bool from_raw = ex_ == data_eid && raw_in.dtype == CVMK_I8 && cvmk_stem_pack_supported(&sp) &&
                            !dev_env("CVM_B200_NO_STEM_PACK");
      if (from_raw) {  // gather straight from the NCHW input: no channels-last copy of it is needed
        add_step(label + "[stem_pack]", [sp](cudaStream_t s) { return cvmk_stem_pack(&sp, s); });
      }
      DevBuf xin_holder;
      if (!from_raw) xin_holder = materialize(ex_);
      const DevBuf& xin = xin_holder;
      cvmk_im2col_desc pk;
      memset(&pk, 0, sizeof(pk));
      pk.x = (const int8_t*)xin.ptr; pk.a = amat;
      pk.N = N; pk.H = H; pk.W = W; pk.C = C; pk.KH = KH; pk.KW = KW; pk.OH = OH; pk.OW = OW;
      pk.stride_h = sh; pk.stride_w = sw; pk.pad_h = ph; pk.pad_w = pw; pk.dil_h = dh; pk.dil_w = dw;
      pk.Kp = kp;
      if (!from_raw) add_step(label + "[pack]", [pk](cudaStream_t s) { return cvmk_im2col_pack(&pk, s); });
      cvmk_conv_desc d = packed;
      d.x = amat; d.w = wdev; d.y = out.ptr; d.y_dtype = out.dtype;
      d.status = ex.status_dev_;
      d.ep = ch.ep;
      void* mem = nullptr;
      CHECK(posix_memalign(&mem, 64, sizeof(cvmk_conv_plan)) == 0);
      ex.plans_.emplace_back((cvmk_conv_plan*)mem, plan_deleter);
      cvmk_conv_plan* plan = ex.plans_.back().get();
      KERNEL_OK(cvmk_conv2d_tc_prepare(&d, plan));
      add_step(label + "[tc]", [plan](cudaStream_t s) { return cvmk_conv2d_tc_launch(plan, s); });
      return;
    }

    if (tc_pad) {
      DevBuf xin = i8_view(ex_, label);
      DevBuf tmp = out;
      tmp.shape = Shape{(int64_t)N, (int64_t)OCp, (int64_t)OH, (int64_t)OW};
      tmp.nhwc = true;
      tmp.ptr = act_alloc(tmp.bytes());
      cvmk_conv_desc d = probe;
      d.OC = OCp;
      d.x = (const int8_t*)xin.ptr; d.w = wdev; d.y = tmp.ptr; d.y_dtype = tmp.dtype;
      d.status = ex.status_dev_;
      d.ep = ch.ep;
      void* mem = nullptr;
      CHECK(posix_memalign(&mem, 64, sizeof(cvmk_conv_plan)) == 0);
      ex.plans_.emplace_back((cvmk_conv_plan*)mem, plan_deleter);
      cvmk_conv_plan* plan = ex.plans_.back().get();
      KERNEL_OK(cvmk_conv2d_tc_prepare(&d, plan));
      add_step(label + "[tc]", [plan](cudaStream_t s) { return cvmk_conv2d_tc_launch(plan, s); });
      const auto ss = phys_strides(tmp.shape, true), ds = phys_strides(out.shape, out.nhwc);
      std::vector<GDim> dims;
      for (int k = 0; k < 4; ++k) dims.push_back({out.shape[k], ss[k], ds[k]});
      emit_gather(tmp, 0, out, dims, label + ":channels");
      return;
    }

    if (tc) {
      DevBuf xin = i8_view(ex_, label);
      cvmk_conv_desc d = probe;
      d.x = (const int8_t*)xin.ptr; d.w = wdev; d.y = out.ptr; d.y_dtype = out.dtype;
      d.status = ex.status_dev_;
      d.ep = ch.ep;
      // Narrow 1x1 layers (few input and output channels) make tiles with one or two tensor-core
      // instructions each, and what a tile costs beside them dominates.  f neighbouring pixels of
      // an NHWC tensor are f * C contiguous bytes, so the same layer is also [M / f, f * C] x
      // block-diagonal weights [f * OC, f * C] -> [M / f, f * OC], byte for byte the same output:
      // f times the multiplies (zeros), 1 / f of the tiles.  32 -> 64 channels at 112 x 112, batch
      // 256: 0.116 -> 0.058 ms with f = 4; 64 -> 64 at 56 x 56: 0.032 -> 0.022 ms with f = 2.
      int fold = 1;
      const std::vector<Range> parts = batch_ranges(N);
      if (!dense && groups == 1 && KH == 1 && KW == 1 && sh == 1 && sw == 1 && ph == 0 && pw == 0 &&
          xin.nhwc && out.nhwc && (!use_bias || g.params.count(g.entry_id(n.inputs[2])) > 0) &&
          !dev_env("CVM_B200_NO_PIXEL_FOLD")) {
        auto whole = [&](int f) {   // every part of the batch is a whole number of folded pixels
          for (const Range& r : parts)
            if (r.begin * OH * OW % f != 0) return false;
          return (int64_t)N * OH * OW % f == 0;
        };
        while (fold < 4 && 2 * fold * C <= 128 && 2 * fold * OC <= 256 && whole(2 * fold)) fold *= 2;
      }
      if (fold > 1) {
        const int Cf = fold * C, OCf = fold * OC;
        std::vector<int8_t> wf((size_t)OCf * Cf, 0);   // block j: rows j * OC .., columns j * C ..
        for (int j = 0; j < fold; ++j)
          for (int o = 0; o < OC; ++o)
            memcpy(&wf[((size_t)(j * OC + o)) * Cf + (size_t)j * C], &w8[(size_t)o * C], (size_t)C);
        int8_t* wfdev = (int8_t*)ex.dalloc(wf.size());
        CUDA_OK(cudaMemcpy(wfdev, wf.data(), wf.size(), cudaMemcpyHostToDevice));
        d.w = wfdev;
        if (use_bias) {   // the bias once per folded pixel
          const auto& bv = g.params.find(g.entry_id(n.inputs[2]))->second.data;
          std::vector<int32_t> bf((size_t)(OCf + 31) / 32 * 32, 0);
          for (int j = 0; j < fold; ++j)
            for (int o = 0; o < OC; ++o) bf[(size_t)j * OC + o] = bv[o];
          int32_t* bfdev = (int32_t*)ex.dalloc(bf.size() * 4);
          CUDA_OK(cudaMemcpy(bfdev, bf.data(), bf.size() * 4, cudaMemcpyHostToDevice));
          d.ep.s[0].ptr = bfdev;
        }
        d.N = (int32_t)((int64_t)N * OH * OW / fold);
        d.H = d.W = d.OH = d.OW = 1;
        d.C = Cf; d.OC = OCf;
      }
      void* mem = nullptr;
      CHECK(posix_memalign(&mem, 64, sizeof(cvmk_conv_plan)) == 0);
      ex.plans_.emplace_back((cvmk_conv_plan*)mem, plan_deleter);
      cvmk_conv_plan* plan = ex.plans_.back().get();
      KERNEL_OK(cvmk_conv2d_tc_prepare(&d, plan));
      add_step(label + "[tc]", [plan](cudaStream_t s) { return cvmk_conv2d_tc_launch(plan, s); });
      // The parts of the batch (every operand is batch-major, so a part is a contiguous slice).
      if (xin.nhwc && out.nhwc) {
        ex.steps_.back().images = N;
        const int64_t per_image = fold > 1 ? (int64_t)OH * OW : 1;   // (folded pixels: d.N counts fold-th parts of pixels)
        // (every part's operands start on 16 bytes: odd images of 8 or 24 channels do not)
        bool aligned = true;
        for (const Range& r : parts) {
          const size_t out_first = (size_t)(r.begin * per_image / fold) * d.OH * d.OW * d.OC;
          aligned &= out_first * d.y_dtype % 16 == 0;
          for (int i = 0; i < d.ep.n; ++i) {
            const cvmk_ep_step& st = d.ep.s[i];
            if ((st.op == CVMK_EP_ADD_T || st.op == CVMK_EP_SUB_T || st.op == CVMK_EP_RSUB_T) && st.ptr) aligned &= out_first * st.ptr_dtype % 16 == 0;
          }
        }
        for (const Range& r : aligned ? parts : std::vector<Range>()) {
          const size_t first = (size_t)(r.begin * per_image / fold);
          cvmk_conv_desc cd = d;
          cd.N = (int)((r.end - r.begin) * per_image / fold);
          const size_t out_first = first * d.OH * d.OW * d.OC;
          cd.x = d.x + first * d.H * d.W * d.C;
          cd.y = (char*)d.y + out_first * d.y_dtype;
          for (int i = 0; i < cd.ep.n; ++i) {
            cvmk_ep_step& st = cd.ep.s[i];
            if ((st.op == CVMK_EP_ADD_T || st.op == CVMK_EP_SUB_T || st.op == CVMK_EP_RSUB_T) && st.ptr)
              st.ptr = (const char*)st.ptr + out_first * st.ptr_dtype;
          }
          ex.steps_.back().chunk.push_back(part_launch(cd, cvmk_conv2d_tc_prepare, cvmk_conv2d_tc_launch));
        }
      }
    } else {
      DevBuf& xin = materialize(ex_);
      cvmk_conv_direct_desc d;
      memset(&d, 0, sizeof(d));
      d.x = xin.ptr; d.x_dtype = xin.dtype; d.narrow_x = groups == 1;
      d.w = wdev; d.y = out.ptr; d.y_dtype = out.dtype;
      d.N = N; d.H = H; d.W = W; d.C = C; d.OC = OC; d.KH = KH; d.KW = KW; d.OH = OH; d.OW = OW; d.groups = groups;
      d.stride_h = sh; d.stride_w = sw; d.pad_h = ph; d.pad_w = pw; d.dil_h = dh; d.dil_w = dw;
      d.depthwise = depthwise;
      d.acc_bound = probe.acc_bound;
      d.bias_static = probe.bias_static;
      d.status = ex.status_dev_;
      d.ep = ch.ep;
      add_step(label + (depthwise ? "[dw]" : "[direct]"), [d](cudaStream_t s) { return cvmk_conv2d_direct(&d, s); });
      // The parts of the batch (batch-major operands: a part is a contiguous slice).
      ex.steps_.back().images = d.N;
      for (const Range& r : xin.nhwc && out.nhwc ? batch_ranges(d.N) : std::vector<Range>()) {
        cvmk_conv_direct_desc cd = d;
        const size_t out_first = (size_t)r.begin * d.OH * d.OW * d.OC;
        cd.N = (int)(r.end - r.begin);
        cd.x = (const char*)d.x + (size_t)r.begin * d.H * d.W * d.C * d.x_dtype;
        cd.y = (char*)d.y + out_first * d.y_dtype;
        for (int i = 0; i < cd.ep.n; ++i) {
          cvmk_ep_step& st = cd.ep.s[i];
          if ((st.op == CVMK_EP_ADD_T || st.op == CVMK_EP_SUB_T || st.op == CVMK_EP_RSUB_T) && st.ptr)
            st.ptr = (const char*)st.ptr + out_first * st.ptr_dtype;
        }
        ex.steps_.back().chunk.push_back([cd](cudaStream_t s) { return cvmk_conv2d_direct(&cd, s); });
      }
    }
  }

  // Element-wise root: unary ops, elemwise_add/sub, broadcast with a scalar parameter.
  bool lower_elemwise_root(uint32_t nid) {
    const Node& n = g.nodes[nid];
    uint32_t src = g.entry_id(n.inputs[0]);
    cvmk_ep_step st;
    if (!node_as_step(nid, src, &st)) {
      if (n.inputs.size() == 2) {
        src = g.entry_id(n.inputs[1]);
        if (!node_as_step(nid, src, &st)) return false;
      } else {
        return false;
      }
    }
    if (g.shape[src] != g.shape[g.entry_id(nid, 0)]) return false;
    Chain ch;
    memset(&ch.ep, 0, sizeof(ch.ep));
    ch.ep.s[0] = st;
    ch.ep.n = 1;
    ch.tail_eid = g.entry_id(nid, 0);
    ch.tail_nid = nid;
    extend_chain(&ch);
    bind_chain(&ch.ep);
    const DevBuf x = materialize(src);
    const DevBuf y = materialize(ch.tail_eid);
    const cvmk_epilogue ep = ch.ep;
    const int64_t cnt = shape_size(x.shape);
    add_step(n.op->name + ":" + n.name(), [x, y, ep, cnt](cudaStream_t s) {
      return cvmk_elemwise(x.ptr, x.dtype, y.ptr, y.dtype, cnt, &ep, s);
    });
    return true;
  }

  void lower_broadcast(uint32_t nid) {
    const Node& n = g.nodes[nid];
    const std::string& op = n.op->name;
    const uint32_t ea = g.entry_id(n.inputs[0]), eb = g.entry_id(n.inputs[1]), eo = g.entry_id(nid, 0);
    const DevBuf a = materialize(ea), b = materialize(eb);
    Chain ch;
    memset(&ch.ep, 0, sizeof(ch.ep));
    ch.tail_eid = eo;
    ch.tail_nid = nid;
    // A fused tail must keep the shape (and with it the layout) of this node's output.
    extend_chain(&ch);
    bind_chain(&ch.ep);
    const DevBuf y = materialize(ch.tail_eid);
    cvmk_strided_desc d;
    memset(&d, 0, sizeof(d));
    d.op = (op == "broadcast_add" || op == "elemwise_add") ? CVMK_OP_ADD
         : (op == "broadcast_sub" || op == "elemwise_sub") ? CVMK_OP_SUB
         : op == "broadcast_mul" ? CVMK_OP_MUL : op == "broadcast_max" ? CVMK_OP_MAX
         : op == "broadcast_div" ? CVMK_OP_DIV : CVMK_OP_GREATER;
    const Shape& os = y.shape;
    const auto order = phys_order(os, y.nhwc);
    const auto ys = phys_strides(os, y.nhwc);
    const auto as = phys_strides(a.shape, a.nhwc), bs = phys_strides(b.shape, b.nhwc);
    d.ndim = (int)os.size();
    const int offa = (int)os.size() - (int)a.shape.size(), offb = (int)os.size() - (int)b.shape.size();
    for (int k = 0; k < d.ndim; ++k) {
      const int j = order[k];
      d.extent[k] = os[j];
      d.y_stride[k] = ys[j];
      d.a_stride[k] = (j - offa >= 0 && a.shape[j - offa] != 1) ? as[j - offa] : 0;
      d.b_stride[k] = (j - offb >= 0 && b.shape[j - offb] != 1) ? bs[j - offb] : 0;
    }
    d.a = a.ptr; d.a_dtype = a.dtype; d.b = b.ptr; d.b_dtype = b.dtype; d.y = y.ptr; d.y_dtype = y.dtype;
    d.ep = ch.ep;
    add_step(op + ":" + n.name(), [d](cudaStream_t s) { return cvmk_strided(&d, s); });
  }

  void lower_pool(uint32_t nid) {
    const Node& n = g.nodes[nid];
    const uint32_t ei = g.entry_id(n.inputs[0]), eo = g.entry_id(nid, 0);
    const DevBuf x = materialize(ei);
    const DevBuf y = materialize(eo);
    CHECK(x.dtype == y.dtype);
    const Shape& pad = n.attrs.t("padding");
    cvmk_pool_desc d;
    memset(&d, 0, sizeof(d));
    d.x = x.ptr; d.y = y.ptr; d.dtype = x.dtype;
    d.N = (int)x.shape[0]; d.C = (int)x.shape[1]; d.H = (int)x.shape[2]; d.W = (int)x.shape[3];
    d.OH = (int)y.shape[2]; d.OW = (int)y.shape[3];
    d.KH = (int)n.attrs.t("pool_size")[0]; d.KW = (int)n.attrs.t("pool_size")[1];
    d.stride_h = (int)n.attrs.t("strides")[0]; d.stride_w = (int)n.attrs.t("strides")[1];
    d.pad_h = (int)pad[0]; d.pad_w = (int)(pad.size() == 2 ? pad[1] : pad[0]);
    add_step("max_pool2d:" + n.name(), [d](cudaStream_t s) { return cvmk_max_pool2d(&d, s); });
    ex.steps_.back().images = d.N;
    for (const Range& r : x.nhwc && y.nhwc ? batch_ranges(d.N) : std::vector<Range>()) {
      cvmk_pool_desc cd = d;
      cd.N = (int)(r.end - r.begin);
      cd.x = (const char*)d.x + (size_t)r.begin * d.H * d.W * d.C * d.dtype;
      cd.y = (char*)d.y + (size_t)r.begin * d.OH * d.OW * d.C * d.dtype;
      ex.steps_.back().chunk.push_back([cd](cudaStream_t s) { return cvmk_max_pool2d(&cd, s); });
    }
  }

  void lower_upsampling(uint32_t nid) {
    const Node& n = g.nodes[nid];
    const DevBuf x = materialize(g.entry_id(n.inputs[0]));
    const DevBuf y = materialize(g.entry_id(nid, 0));
    const int64_t sc = n.attrs.i("scale");
    const int64_t N = x.shape[0], C = x.shape[1], H = x.shape[2], W = x.shape[3];
    const auto xs = phys_strides(x.shape, x.nhwc), ys = phys_strides(y.shape, y.nhwc);
    cvmk_strided_desc d;
    memset(&d, 0, sizeof(d));
    d.op = CVMK_OP_COPY;
    d.ndim = 6;
    // iteration space (N, H, s, W, s, C); the two s extents do not move the source
    const int64_t ext[6] = {N, H, sc, W, sc, C};
    const int64_t as[6] = {xs[0], xs[2], 0, xs[3], 0, xs[1]};
    const int64_t yst[6] = {ys[0], ys[2] * sc, ys[2], ys[3] * sc, ys[3], ys[1]};
    for (int k = 0; k < 6; ++k) { d.extent[k] = ext[k]; d.a_stride[k] = as[k]; d.y_stride[k] = yst[k]; }
    d.a = x.ptr; d.a_dtype = x.dtype; d.y = y.ptr; d.y_dtype = y.dtype;
    add_step("upsampling:" + n.name(), [d](cudaStream_t s) { return cvmk_strided(&d, s); });
  }

  void lower_concat(uint32_t nid) {
    const Node& n = g.nodes[nid];
    const DevBuf y = materialize(g.entry_id(nid, 0));
    const int nd = (int)y.shape.size();
    int axis = (int)n.attrs.i("axis");
    if (axis < 0) axis += nd;
    const auto ys = phys_strides(y.shape, y.nhwc);
    int64_t offset = 0;
    std::vector<cvmk_strided_desc> all;
    for (size_t m = 0; m < n.inputs.size(); ++m) {
      const DevBuf x = materialize(g.entry_id(n.inputs[m]));
      const auto order = phys_order(x.shape, y.nhwc);
      const auto xs = phys_strides(x.shape, x.nhwc);
      cvmk_strided_desc d;
      memset(&d, 0, sizeof(d));
      d.op = CVMK_OP_COPY;
      d.ndim = nd;
      for (int k = 0; k < nd; ++k) {
        d.extent[k] = x.shape[order[k]];
        d.a_stride[k] = xs[order[k]];
        d.y_stride[k] = ys[order[k]];
      }
      d.a = x.ptr; d.a_dtype = x.dtype; d.y = y.ptr; d.y_dtype = y.dtype;
      d.y_off = offset * ys[axis];
      offset += x.shape[axis];
      all.push_back(d);
    }
    // all inputs in one launch when they move whole vectors, else one launch each
    add_step("concatenate:" + n.name(), [all](cudaStream_t s) { return cvmk_strided_batch(all.data(), (int32_t)all.size(), s); });
  }

  // flatten / reshape / squeeze / expand_dims: the row-major element order is preserved.
  void lower_reshape(uint32_t nid) {
    const Node& n = g.nodes[nid];
    const uint32_t ei = g.entry_id(n.inputs[0]), eo = g.entry_id(nid, 0);
    DevBuf src = canon_view(ei, n.op->name + ":" + n.name());
    DevBuf& out = buf[eo];
    CHECK(out.dtype == src.dtype);
    if (!out.nhwc) {
      out.ptr = src.ptr;  // alias
      return;
    }
    materialize(eo);
    DevBuf as_canon = out;
    as_canon.nhwc = false;
    as_canon.ptr = src.ptr;
    emit_convert(as_canon, out, n.op->name + ":" + n.name() + ":to_nhwc");
  }

  // sum / max.  The kept-dimension mapping follows cpu/ops/reduce.cc:66-89 literally, including
  // its pairing of the output's non-unit dimensions with the input's non-reduced ones from the
  // right.
  void lower_reduce(uint32_t nid) {
    const Node& n = g.nodes[nid];
    const uint32_t ei = g.entry_id(n.inputs[0]), eo = g.entry_id(nid, 0);
    DevBuf x = materialize(ei);
    const Shape xs = x.shape;
    const Shape& ysh = g.shape[eo];
    const int xnd = (int)xs.size();
    Shape axis = n.attrs.t("axis");
    const bool exclude = n.attrs.b("exclude");
    for (auto& a : axis) if (a < 0) a += xnd;
    std::vector<int64_t> real;
    if (!exclude) real.assign(axis.begin(), axis.end());
    else {
      for (int i = 0; i < xnd; ++i)
        if (std::find(axis.begin(), axis.end(), i) == axis.end()) real.push_back(i);
    }
    Chain ch;
    memset(&ch.ep, 0, sizeof(ch.ep));
    ch.tail_eid = eo;
    ch.tail_nid = nid;
    const std::string label = n.op->name + ":" + n.name();
    if (exclude && real.empty()) {  // plain copy, reduce.cc:38-39
      extend_chain(&ch);
      bind_chain(&ch.ep);
      DevBuf y = materialize(ch.tail_eid);
      DevBuf srcv = x;
      srcv.shape = y.shape;  // same element order when both are row-major
      if (x.nhwc || y.nhwc) {
        DevBuf c = canon_view(ei, label);
        c.shape = y.shape;
        emit_convert(c, y, label, &ch.ep);
      } else {
        emit_convert(srcv, y, label, &ch.ep);
      }
      return;
    }
    const bool out_needs_convert = wants_nhwc(ysh);
    if (!out_needs_convert) { extend_chain(&ch); bind_chain(&ch.ep); }
    // The reference pairs the output's non-unit dimensions with the input's kept ones from the
    // right and steps by row-major strides (reduce.cc:66-89).  When unit dimensions make the
    // pairing land on a dimension of another extent, the walk leaves that dimension and carries
    // into its neighbours; only the row-major layout reproduces that, so such inputs are read
    // from a row-major copy.
    if (x.nhwc && !real.empty()) {
      std::vector<char> fl(xnd, 0);
      for (auto a : real) fl[a] = 1;
      std::vector<int64_t> nz;
      for (auto v : ysh) if (v != 1) nz.push_back(v);
      bool straight = true;
      int xj = xnd - 1;
      for (int j = (int)nz.size() - 1; j >= 0; --j) {
        while (xj >= 0 && fl[xj--]) {}
        straight &= xj + 1 >= 0 && xj + 1 < xnd && xs[xj + 1] == nz[j];
      }
      if (!straight) x = canon_view(ei, label);
    }
    const auto xst = phys_strides(xs, x.nhwc);
    cvmk_reduce_desc d;
    memset(&d, 0, sizeof(d));
    d.is_max = n.op->name == "max";
    if (real.empty()) {
      d.init_zero = 1;
      d.n_keep = 0;
      d.n_red = xnd;
      for (int k = 0; k < xnd; ++k) { d.red_extent[k] = xs[k]; d.red_stride[k] = xst[k]; }
    } else {
      std::vector<char> flag(xnd, 0);
      for (auto a : real) flag[a] = 1;
      std::sort(real.begin(), real.end());
      d.n_red = (int)real.size();
      for (int k = 0; k < d.n_red; ++k) { d.red_extent[k] = xs[real[k]]; d.red_stride[k] = xst[real[k]]; }
      // every_xdim_size of the reference is the row-major stride; here the physical one is used,
      // which addresses the same logical element.
      std::vector<int64_t> ynz;
      for (auto v : ysh) if (v != 1) ynz.push_back(v);
      d.n_keep = (int)ynz.size();
      int xj = xnd - 1;
      for (int j = d.n_keep - 1; j >= 0; --j) {
        while (xj >= 0 && flag[xj--]) {}
        d.keep_extent[j] = ynz[j];
        d.keep_stride[j] = xj + 1 >= 0 && xj + 1 < xnd ? xst[xj + 1] : 0;
      }
    }
    d.x = x.ptr; d.x_dtype = x.dtype;
    if (out_needs_convert) {
      DevBuf tmp = buf[eo];
      tmp.nhwc = false;
      tmp.ptr = act_alloc(tmp.bytes());
      d.y = tmp.ptr; d.y_dtype = tmp.dtype;
      add_step(label, [d](cudaStream_t s) { return cvmk_reduce(&d, s); });
      emit_convert(tmp, materialize(eo), label + ":to_nhwc");
    } else {
      DevBuf y = materialize(ch.tail_eid);
      d.y = y.ptr; d.y_dtype = y.dtype;
      d.ep = ch.ep;
      add_step(label, [d](cudaStream_t s) { return cvmk_reduce(&d, s); });
    }
  }

  // ------------------------------------------------------------------ index-map transforms
  // One dimension of a gather: `extent` points, each moving the source by a_stride and the
  // destination by y_stride elements.
  struct GDim { int64_t extent, a_stride, y_stride; };

  // dst[y_off + sum c_k ys_k] = src[a_off + sum c_k as_k] as strided copies.  Unit extents are
  // dropped, the destination order decides the iteration order (coalesced writes), neighbours
  // that form one run in both tensors are merged, and spaces of more than six extents are
  // peeled into several launches.
  void emit_gather(const DevBuf& src, int64_t a_off, const DevBuf& dst, std::vector<GDim> dims,
                   const std::string& label) {
    std::vector<GDim> v;
    for (const auto& d : dims) if (d.extent != 1) v.push_back(d);
    std::stable_sort(v.begin(), v.end(), [](const GDim& a, const GDim& b) { return a.y_stride > b.y_stride; });
    std::vector<GDim> m;
    for (const auto& d : v) {
      if (!m.empty() && m.back().a_stride == d.a_stride * d.extent && m.back().y_stride == d.y_stride * d.extent) {
        m.back().extent *= d.extent;
        m.back().a_stride = d.a_stride;
        m.back().y_stride = d.y_stride;
      } else {
        m.push_back(d);
      }
    }
    if (m.empty()) m.push_back({1, 0, 0});
    emit_gather_peeled(src, a_off, dst, 0, m, label);
  }
  void emit_gather_peeled(const DevBuf& src, int64_t a_off, const DevBuf& dst, int64_t y_off,
                          const std::vector<GDim>& m, const std::string& label) {
    if (m.size() > 6) {
      std::vector<GDim> rest(m.begin() + 1, m.end());
      for (int64_t c = 0; c < m[0].extent; ++c)
        emit_gather_peeled(src, a_off + c * m[0].a_stride, dst, y_off + c * m[0].y_stride, rest, label);
      return;
    }
    cvmk_strided_desc d;
    memset(&d, 0, sizeof(d));
    d.op = CVMK_OP_COPY;
    d.ndim = (int)m.size();
    for (int k = 0; k < d.ndim; ++k) {
      d.extent[k] = m[k].extent;
      d.a_stride[k] = m[k].a_stride;
      d.y_stride[k] = m[k].y_stride;
    }
    d.a = src.ptr; d.a_dtype = src.dtype; d.a_off = a_off;
    d.y = dst.ptr; d.y_dtype = dst.dtype; d.y_off = y_off;
    add_step(label, [d](cudaStream_t s) { return cvmk_strided(&d, s); });
  }

  // transpose / strided_slice / slice_like / repeat / tile (cpu/ops/ops.cc:603-683, :743-866):
  // every output element is one input element, at an index that is affine in the output index.
  void lower_index_map(uint32_t nid) {
    const Node& n = g.nodes[nid];
    const std::string& op = n.op->name;
    const DevBuf x = materialize(g.entry_id(n.inputs[0]));
    if (transpose_is_identity(nid) && !dev_env("CVM_B200_NO_TRANSPOSE_ALIAS")) {
      DevBuf& out = buf[g.entry_id(nid, 0)];
      bool written = false;   // an entry that non_max_suppression overwrites in place keeps its own memory
      for (const auto& wv : input_writers) written |= wv.second == g.entry_id(nid, 0) || wv.second == g.entry_id(n.inputs[0]);
      if (!out.ptr && !out.nhwc && out.dtype == x.dtype && !written) {
        out.ptr = x.ptr;  // alias
        return;
      }
    }
    const DevBuf y = materialize(g.entry_id(nid, 0));
    const Shape &xsh = x.shape, &ysh = y.shape;
    const auto xs = phys_strides(xsh, x.nhwc), ys = phys_strides(ysh, y.nhwc);
    const int xnd = (int)xsh.size(), ynd = (int)ysh.size();
    std::vector<GDim> dims;
    int64_t a_off = 0;
    if (op == "transpose") {
      Shape axes = n.attrs.t("axes");
      for (int j = 0; j < ynd; ++j) {
        int64_t ax = axes.empty() ? ynd - 1 - j : axes[j];
        if (ax < 0) ax += xnd;
        dims.push_back({ysh[j], xs[ax], ys[j]});
      }
    } else if (op == "strided_slice") {
      Shape b = n.attrs.t("begin"), st = n.attrs.t("stride");
      for (int i = (int)b.size(); i < xnd; ++i) b.push_back(0);
      for (int i = (int)st.size(); i < xnd; ++i) st.push_back(1);
      for (int j = 0; j < xnd; ++j) {
        const int64_t lo = st[j] < 0 ? -1 : 0, hi = st[j] < 0 ? xsh[j] - 1 : xsh[j];
        int64_t bg = b[j] < 0 ? b[j] + xsh[j] : b[j];
        bg = std::min(std::max(bg, lo), hi);
        a_off += bg * xs[j];
        dims.push_back({ysh[j], xs[j] * st[j], ys[j]});
      }
    } else if (op == "slice_like") {
      for (int j = 0; j < xnd; ++j) dims.push_back({ysh[j], xs[j], ys[j]});
    } else if (op == "repeat") {
      int axis = (int)n.attrs.i("axis");
      if (axis < 0) axis += xnd;
      const int64_t rep = n.attrs.i("repeats");
      for (int j = 0; j < xnd; ++j) {
        if (j == axis) {
          dims.push_back({xsh[j], xs[j], ys[j] * rep});
          dims.push_back({rep, 0, ys[j]});
        } else {
          dims.push_back({ysh[j], xs[j], ys[j]});
        }
      }
    } else {  // tile: right-aligned, output column c reads input column c % extent
      for (int j = 0; j < ynd; ++j) {
        const int xj = j - (ynd - xnd);
        if (xj < 0) {
          dims.push_back({ysh[j], 0, ys[j]});
        } else {
          dims.push_back({ysh[j] / xsh[xj], 0, ys[j] * xsh[xj]});
          dims.push_back({xsh[xj], xs[xj], ys[j]});
        }
      }
    }
    emit_gather(x, a_off, y, dims, op + ":" + n.name());
  }

  // A row-major buffer to produce entry `eid` into; finish_rowmajor() moves it into the entry's
  // own layout when that is channels-last.
  DevBuf rowmajor_target(uint32_t eid) {
    DevBuf& b = materialize(eid);
    if (!b.nhwc) return b;
    DevBuf t = b;
    t.nhwc = false;
    t.ptr = act_alloc(t.bytes());
    return t;
  }
  void finish_rowmajor(const DevBuf& t, uint32_t eid, const std::string& label) {
    if (t.ptr != buf[eid].ptr) emit_convert(t, buf[eid], label + ":to_nhwc");
  }

  // take (cpu/ops/ops.cc:868-945) and cvm_lut (:947-956)
  void lower_take(uint32_t nid) {
    const Node& n = g.nodes[nid];
    const bool lut = n.op->name == "cvm_lut";
    const std::string label = n.op->name + ":" + n.name();
    const uint32_t e_x = g.entry_id(n.inputs[lut ? 1 : 0]), e_i = g.entry_id(n.inputs[lut ? 0 : 1]);
    const uint32_t eo = g.entry_id(nid, 0);
    cvmk_take_desc d;
    memset(&d, 0, sizeof(d));
    const DevBuf x = canon_view(e_x, label);
    d.x = x.ptr; d.x_dtype = x.dtype;
    if (lut || !n.attrs.has.at("axis")) {
      d.outer = 1; d.inner = 1;
      d.extent = shape_size(x.shape);
    } else {
      int axis = (int)n.attrs.i("axis");
      if (axis < 0) axis += (int)x.shape.size();
      d.outer = d.inner = 1;
      for (int j = 0; j < axis; ++j) d.outer *= x.shape[j];
      for (int j = axis + 1; j < (int)x.shape.size(); ++j) d.inner *= x.shape[j];
      d.extent = x.shape[axis];
    }
    d.count = shape_size(g.shape[e_i]);
    if (lut) {
      // flat lookup: the output has the shape, and therefore the layout, of the index tensor
      const DevBuf idx = materialize(e_i);
      const DevBuf y = materialize(eo);
      d.indices = idx.ptr; d.idx_dtype = idx.dtype; d.y = y.ptr; d.y_dtype = y.dtype;
      add_step(label, [d](cudaStream_t s) { return cvmk_take(&d, s); });
      return;
    }
    const DevBuf idx = canon_view(e_i, label + ":indices");
    const DevBuf y = rowmajor_target(eo);
    d.indices = idx.ptr; d.idx_dtype = idx.dtype; d.y = y.ptr; d.y_dtype = y.dtype;
    add_step(label, [d](cudaStream_t s) { return cvmk_take(&d, s); });
    finish_rowmajor(y, eo, label);
  }

  // where (cpu/ops/ops.cc:1049-1075).  x, y and the result share a shape, hence a layout; a
  // condition of that shape does too, and a 1-D condition indexes the outermost dimension, which is
  // outermost in both layouts.
  void lower_where(uint32_t nid) {
    const Node& n = g.nodes[nid];
    const DevBuf c = materialize(g.entry_id(n.inputs[0]));
    const DevBuf x = materialize(g.entry_id(n.inputs[1]));
    const DevBuf y = materialize(g.entry_id(n.inputs[2]));
    const DevBuf o = materialize(g.entry_id(nid, 0));
    cvmk_where_desc d;
    memset(&d, 0, sizeof(d));
    d.cond = c.ptr; d.cond_dtype = c.dtype;
    d.x = x.ptr; d.x_dtype = x.dtype;
    d.y = y.ptr; d.y_dtype = y.dtype;
    d.out = o.ptr; d.out_dtype = o.dtype;
    d.n = shape_size(x.shape);
    d.inner = c.shape.size() == x.shape.size() ? 1 : d.n / x.shape[0];
    add_step("where:" + n.name(), [d](cudaStream_t s) { return cvmk_where(&d, s); });
  }

  void lower_gvc(uint32_t nid) {
    const Node& n = g.nodes[nid];
    const std::string label = "get_valid_counts:" + n.name();
    const uint32_t in_eid = g.entry_id(n.inputs[0]);
    // Rows that are the network input, read by nobody else: the operator reads the uploaded bytes
    // and applies the input clamp itself, instead of a copy of the whole tensor doing it first.
    const bool from_raw = in_eid == data_eid && raw_in.dtype == CVMK_I32 && uses[in_eid] == 1 && !is_head[in_eid] &&
                          !buf[in_eid].ptr && !dev_env("CVM_B200_NO_GVC_FROM_INPUT");
    const DevBuf x = from_raw ? raw_in : canon_i32_view(in_eid, label);
    const int clamp = from_raw ? data_range : 0;
    const DevBuf vc = materialize(g.entry_id(nid, 0));
    const DevBuf y = materialize(g.entry_id(nid, 1));
    CHECK(vc.dtype == CVMK_I32 && y.dtype == CVMK_I32);
    const int B = (int)x.shape[0], N = (int)x.shape[1], K = (int)x.shape[2];
    const int thr = (int)n.attrs.i("score_threshold");
    add_step(label, [x, y, vc, B, N, K, thr, clamp](cudaStream_t s) {
      return cvmk_get_valid_counts_clamped((const int32_t*)x.ptr, (int32_t*)y.ptr, (int32_t*)vc.ptr, B, N, K, thr, clamp, s);
    });
    ex.steps_.back().from_input = from_raw;
    ex.steps_.back().images = B;
    const std::vector<Range> parts = from_raw ? batch_ranges(B) : std::vector<Range>();
    input_ranges(parts, (size_t)N * K * 4);
    for (const Range& r : parts) {   // while later images upload
      const int64_t b0 = r.begin, rows = b0 * N * K;
      const int count = (int)(r.end - b0);
      ex.steps_.back().chunk.push_back([x, y, vc, b0, rows, count, N, K, thr, clamp](cudaStream_t s) {
        return cvmk_get_valid_counts_clamped((const int32_t*)x.ptr + rows, (int32_t*)y.ptr + rows, (int32_t*)vc.ptr + b0, count, N, K, thr, clamp, s);
      });
    }
  }

  // Outputs of non_max_suppression that hold at most so many bytes of rows per image: images, bytes,
  // device array of the valid counts.
  struct Limited { size_t images, live_bytes; const int32_t* valid_count; };
  std::map<uint32_t, Limited> limited;

  void lower_nms(uint32_t nid) {
    const Node& n = g.nodes[nid];
    const std::string label = "non_max_suppression:" + n.name();
    const DevBuf x = canon_i32_view(g.entry_id(n.inputs[0]), label);
    const DevBuf vc = canon_i32_view(g.entry_id(n.inputs[1]), label);
    const DevBuf y = materialize(g.entry_id(nid, 0));
    CHECK(y.dtype == CVMK_I32);
    cvmk_nms_desc d;
    memset(&d, 0, sizeof(d));
    d.x = (const int32_t*)x.ptr; d.valid_count = (const int32_t*)vc.ptr; d.y = (int32_t*)y.ptr;
    d.B = (int)x.shape[0]; d.N = (int)x.shape[1];
    d.max_output_size = (int)n.attrs.i("max_output_size");
    d.iou_threshold = (int)n.attrs.i("iou_threshold");
    d.top_k = (int)n.attrs.i("top_k");
    d.force_suppress = n.attrs.b("force_suppress") ? 1 : 0;
    d.scratch_bytes = cvmk_nms_scratch_bytes(d.B, d.N);
    d.scratch = act_alloc((size_t)d.scratch_bytes);
    // The CPU operator writes -1 over the input rows outside the top_k (nms.cc:93-97).  That is
    // visible when the input entry is a head or is read again by a later node.
    const uint32_t in_eid = g.entry_id(n.inputs[0]);
    bool observed = false;
    for (const auto& h : g.outputs) observed |= g.entry_id(h) == in_eid;
    for (uint32_t m = nid + 1; m < g.nodes.size(); ++m)
      for (const auto& e : g.nodes[m].inputs) observed |= g.entry_id(e) == in_eid;
    if (observed) {
      const DevBuf own = materialize(in_eid);
      VERIFY(own.ptr == x.ptr) << label << ": its input is read again after the operator, which needs the input "
                               << "stored as int32 rows";
      d.x_writeback = (int32_t*)own.ptr;
    }
    if (d.top_k > 0 && (size_t)d.B * 4 < (size_t)1 << 20) {   // (a small buffer is not shared: the counts stay to the end)
      int64_t bound = std::min<int64_t>(d.N, d.top_k);
      if (d.max_output_size > 0) bound = std::min<int64_t>(bound, d.max_output_size);
      if (bound < d.N) limited[g.entry_id(nid, 0)] = {(size_t)d.B, (size_t)bound * 24, d.valid_count};
    }
    add_step(label, [d](cudaStream_t s) { return cvmk_non_max_suppression(&d, s); });
    ex.steps_.back().images = d.B;
    for (const Range& r : batch_ranges(d.B)) {
      const int first = (int)r.begin, count = (int)(r.end - r.begin);
      ex.steps_.back().chunk.push_back([d, first, count](cudaStream_t s) { return cvmk_non_max_suppression_part(&d, first, count, s); });
    }
  }

  // Lifetimes of the activation buffers in schedule positions (one position per fused group, in
  // the order the groups are launched), then their physical backing.  A buffer is live from the
  // group that first writes it (the group of the producing node, which for a shortcut operand of
  // a fused join can precede the group whose lowering allocated it) to the last group that reads
  // it: the groups of all consumers of every graph entry stored in it (aliases of reshape-like
  // nodes included), the end of the inference for a head.  Reads and writes inside one group all
  // happen at that group's position.  Every kernel launched with programmatic dependent launch
  // waits for the whole preceding kernel before it touches global memory, so a buffer whose last
  // reader sits at position p can be overwritten from position p + 1 on.  The steps that are
  // launched per batch chunk while the input uploads run chunk after chunk, so everything they
  // touch stays live across that whole prefix.
  std::vector<int> step_pos;   // step -> schedule position (-1: before the first group)
  void plan_activations(const std::vector<std::pair<uint32_t, uint32_t>>& order) {
    auto& act = ex.act_;
    if (act.empty()) return;
    const int end = (int)order.size() + 1;
    std::vector<int> pos(g.nodes.size(), -1);
    for (size_t i = 0; i < order.size(); ++i) pos[order[i].second] = (int)i;
    auto group_pos = [&](uint32_t nid) { return root_of[nid] == UINT32_MAX ? -1 : pos[root_of[nid]]; };
    for (auto& a : act) a.first = a.last = pos[a.root];
    auto find = [&](const void* p) -> Executor::ActBuf* {
      for (auto& a : act)
        if ((const char*)p >= (const char*)a.va && (const char*)p < (const char*)a.va + a.va_size) return &a;
      return nullptr;
    };
    std::vector<Executor::ActBuf*> of_entry(g.num_entries, nullptr);
    for (uint32_t nid = 0; nid < g.nodes.size(); ++nid)
      for (uint32_t eid = g.node_row_ptr[nid]; eid < g.node_row_ptr[nid + 1]; ++eid) {
        if (!buf[eid].ptr) continue;
        Executor::ActBuf* a = of_entry[eid] = find(buf[eid].ptr);
        if (!a) continue;
        a->first = std::min(a->first, g.nodes[nid].is_variable() ? -1 : group_pos(nid));
        if (is_head[eid]) a->last = end;
      }
    for (uint32_t nid = 0; nid < g.nodes.size(); ++nid)
      for (const auto& e : g.nodes[nid].inputs)
        if (Executor::ActBuf* a = of_entry[g.entry_id(e)]) a->last = std::max(a->last, group_pos(nid));
    for (auto& a : act) { a.first0 = a.first; a.last0 = a.last; }
    ex.step_pos_ = step_pos;
    // first with the longest prefix that may be chosen; Load() plans again once it is known.  Where the device has
    // no room for that many buffers at once, inferences run without a prefix.
    try {
      ex.PlanForPrefix(ex.prefix_max_);
    } catch (const std::exception&) {
      if (ex.prefix_max_ == 0) throw;
      ex.prefix_max_ = 0;
      ex.PlanForPrefix(0);
    }
  }

  void lower_node(uint32_t nid) {
    const Node& n = g.nodes[nid];
    const std::string& op = n.op->name;
    if (op == "conv2d") return lower_conv_like(nid, false);
    if (op == "dense") return lower_conv_like(nid, true);
    if (op == "max_pool2d") return lower_pool(nid);
    if (op == "upsampling") return lower_upsampling(nid);
    if (op == "concatenate") return lower_concat(nid);
    if (op == "flatten" || op == "reshape" || op == "squeeze" || op == "expand_dims") return lower_reshape(nid);
    if (op == "sum" || op == "max") return lower_reduce(nid);
    if (op == "transpose" || op == "strided_slice" || op == "slice_like" || op == "repeat" || op == "tile")
      return lower_index_map(nid);
    if (op == "take" || op == "cvm_lut") return lower_take(nid);
    if (op == "where") return lower_where(nid);
    if (op == "get_valid_counts") return lower_gvc(nid);
    if (op == "non_max_suppression") return lower_nms(nid);
    if (lower_elemwise_root(nid)) return;
    if (op.compare(0, 10, "broadcast_") == 0 || op == "elemwise_add" || op == "elemwise_sub")
      return lower_broadcast(nid);
    FATAL() << "function undefined cvm.runtime.gpu." << op;
  }

  void run() {
    analyse();
    find_input_writers();
    // graph input: raw API bytes -> clamp to the declared precision -> entry buffer
    int data_nid = -1;
    for (uint32_t nid = 0; nid < g.nodes.size(); ++nid)
      if (g.nodes[nid].is_data()) data_nid = (int)nid;
    CHECK(data_nid >= 0) << "can not find input `data`";
    {
      const uint32_t eid = g.entry_id(data_nid, 0);
      const int prec = g.precision[eid];
      data_eid = eid;
      raw_in.shape = g.shape[eid];
      raw_in.dtype = prec > 8 ? CVMK_I32 : CVMK_I8;
      raw_in.nhwc = false;
      ex.in_bytes_ = raw_in.bytes();
      ex.in_dev_ = ex.dalloc(ex.in_bytes_);
      const size_t padded = (ex.in_bytes_ + 15) & ~(size_t)15;   // (device buffers are whole 256 bytes)
      CUDA_OK(cudaMallocHost(&ex.in_host_, padded));
      memset(ex.in_host_, 0, padded);
      ex.pinned_.push_back(ex.in_host_);
      raw_in.ptr = ex.in_dev_;
      data_range = (int32_t)((1u << (prec - 1)) - 1);
    }
    // Fused groups are emitted at the position of their last member, so every operand of the
    // chain already exists when the kernel runs.
    std::vector<std::pair<uint32_t, uint32_t>> order;  // (schedule position, root)
    {
      // A dry pass decides the groups; the step lists of the groups are then ordered by tail.
      std::vector<std::vector<Step>> per_root(g.nodes.size());
      std::vector<uint32_t> tail(g.nodes.size(), 0);
      root_of.assign(g.nodes.size(), UINT32_MAX);
      std::vector<Step> prologue = ex.steps_;
      ex.steps_.clear();
      for (uint32_t nid = 0; nid < g.nodes.size(); ++nid) {
        const Node& n = g.nodes[nid];
        if (n.is_variable() || absorbed[nid]) continue;
        const size_t before = ex.steps_.size();
        uint32_t last = nid;
        cur_root = nid;
        root_of[nid] = nid;
        lower_node(nid);
        cur_root = UINT32_MAX;
        for (uint32_t k = nid + 1; k < g.nodes.size(); ++k)
          if (absorbed[k] == 1) { absorbed[k] = 2; root_of[k] = nid; last = std::max(last, k); }
        per_root[nid].assign(ex.steps_.begin() + before, ex.steps_.end());
        ex.steps_.resize(before);
        tail[nid] = last;
        order.emplace_back(last, nid);
      }
      std::stable_sort(order.begin(), order.end());
      ex.steps_ = prologue;
      if (buf[data_eid].ptr || is_head[data_eid]) {
        // some consumer reads the input tensor itself: raw API bytes -> clamp to the declared
        // precision (graph_runtime.cc:379-386) -> the entry's own layout
        cvmk_epilogue ep;
        memset(&ep, 0, sizeof(ep));
        ep.n = 1;
        ep.s[0].op = CVMK_EP_CLIP;
        ep.s[0].a = -data_range;
        ep.s[0].b = data_range;
        emit_convert(raw_in, materialize(data_eid), "input:data", &ep);
        Step& st = ex.steps_.back();
        if (!st.chunk.empty()) {
          st.from_input = true;
          input_ranges(batch_ranges(st.images), ex.in_bytes_ / st.images);
        }
      }
      step_pos.assign(ex.steps_.size(), -1);
      for (size_t i = 0; i < order.size(); ++i)
        for (auto& s : per_root[order[i].second]) {
          ex.steps_.push_back(std::move(s));
          step_pos.push_back((int)i);
        }
    }
    // Upload / compute overlap: when the inference starts with a step that takes the input part by
    // part, the leading run of steps that can be cut along the batch may be launched per part.  How
    // much of it is, is decided by measurement after the plan.  Everything the prefix touches is live
    // for all of it (whole-batch buffers, filled part by part), so its length is also a memory
    // decision: ten steps of ResNet-50 at batch 256 hold 1.3 GB, twenty 2.1 GB.
    {
      const size_t cap = 14;
      ex.prefix_max_ = 0;
      if (!ex.range_end_.empty() && !ex.steps_.empty() && ex.steps_[0].from_input)
        while (ex.prefix_max_ < ex.steps_.size() && ex.prefix_max_ < cap && cut_like_first(ex.steps_[ex.prefix_max_])) ++ex.prefix_max_;
    }
    const size_t body = ex.steps_.size();
    plan_activations(order);
    // heads: row-major staging + pinned host mirrors
    for (const auto& e : g.outputs) {
      const uint32_t eid = g.entry_id(e);
      DevBuf c = canon_view(eid, "head");
      HeadOut h;
      h.shape = c.shape;
      h.dtype = c.dtype;
      h.dev = c.ptr;
      h.bytes = c.bytes();
      auto lim = limited.find(eid);
      if (lim != limited.end()) {
        h.images = lim->second.images;
        h.live_bytes = lim->second.live_bytes;
        h.valid_count = lim->second.valid_count;
      }
      CUDA_OK(cudaMallocHost(&h.host, h.bytes));
      ex.pinned_.push_back(h.host);
      ex.heads_.push_back(h);
    }
    // A short graph that can be cut as a whole: the parts of its head leave while later parts compute.
    if (ex.prefix_max_ > 0 && ex.prefix_max_ == body && ex.heads_.size() == 1) {
      if (ex.steps_.size() == body + 1 && cut_like_first(ex.steps_[body])) ++ex.prefix_max_;
      const HeadOut& h = ex.heads_[0];
      const int64_t images = ex.steps_[0].images;
      if (ex.prefix_max_ == ex.steps_.size() && h.shape.size() > 1 && h.shape[0] == images)
        for (const Range& r : batch_ranges(images)) ex.head_range_end_.push_back(h.bytes / images * r.end);
    }
  }
  // (the same number of images: a reshape between two steps may change what a part of the batch is)
  bool cut_like_first(const Step& s) const { return s.chunk.size() == ex.range_end_.size() && s.images == ex.steps_[0].images; }
};

// (a constructor that throws has no destructor: what it had made by then is given back here)
Executor::Executor(const Graph& g, int device_id, int plain_elem_bytes) : g_(g), device_(device_id) {
  try {
    Load(plain_elem_bytes);
  } catch (...) {
    Release();
    throw;
  }
}

void Executor::Load(int plain_elem_bytes) {
  int count = 0;
  CUDA_OK(cudaGetDeviceCount(&count));
  CHECK(device_ >= 0 && device_ < count) << "device_id " << device_ << " out of range (" << count << " GPUs)";
  CUDA_OK(cudaSetDevice(device_));
  CUDA_OK(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
  status_dev_ = (int32_t*)dalloc(256);
  CUDA_OK(cudaMemset(status_dev_, 0, 256));
  CUDA_OK(cudaMallocHost((void**)&status_host_, 256));
  pinned_.push_back(status_host_);
  *status_host_ = 0;
  done_host_ = status_host_ + 32;
  *done_host_ = 0;
  use_graph_ = dev_env("CVM_B200_NO_GRAPH") == nullptr;
  if (vmm().ok && !dev_env("CVM_B200_NO_PLANNER")) {
    const CUmemAllocationProp prop = device_prop(device_);
    size_t gran = 0;
    if (vmm().get_granularity(&gran, &prop, CU_MEM_ALLOC_GRANULARITY_MINIMUM) == CUDA_SUCCESS && gran > 0) {
      vmm_ = true;
      vmm_gran_ = gran;
    }
  }
  Lowering low(*this, g_);
  low.run();
  plain_ = heads_.size() == 1 && heads_[0].dtype == plain_elem_bytes;
  if (!plain_)
    for (auto& h : heads_) h.live_bytes = 0;
  ChooseDownload();
  // One eager pass sets per-kernel attributes and surfaces launch errors before capture.
  Upload(in_host_, stream_);
  Enqueue(stream_);
  CUDA_OK(cudaStreamSynchronize(stream_));
  if (!use_graph_) return;
  if (prefix_max_ > 0) {
    CUDA_OK(cudaStreamCreateWithFlags(&copy_stream_, cudaStreamNonBlocking));
    part_events_.resize(kMaxParts);
    for (auto& e : part_events_) CUDA_OK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  }
  if (!head_range_end_.empty()) {
    CUDA_OK(cudaStreamCreateWithFlags(&down_stream_, cudaStreamNonBlocking));
    part_done_.resize(kMaxParts);
    for (auto& e : part_done_) CUDA_OK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  }
  graph_whole_ = Capture([this] { Enqueue(stream_); });
  ChooseSchedules();
  PlanForPrefix(std::max({from_pinned_.prefix, from_pageable_.prefix, from_device_.prefix}));   // memory for the prefix actually used
  if (in_bytes_ <= kSmallInput)
    graph_staged_ = Capture([this] {
      // (whole 16-byte words whatever the size, see in_host_: 547 215 bytes one by one took 40 us)
      const int64_t padded = ((int64_t)in_bytes_ + 15) & ~(int64_t)15;
      const cvmk_export_segment seg = {in_host_, in_dev_, 1, padded, padded};
      KERNEL_OK(cvmk_export(&seg, 1, stream_));
      Enqueue(stream_);
    });
}

Executor::GraphExec Executor::Capture(const std::function<void()>& enqueue) {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  CUDA_OK(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
  try {
    enqueue();
  } catch (...) {
    if (cudaStreamEndCapture(stream_, &graph) == cudaSuccess) cudaGraphDestroy(graph);
    cudaGetLastError();
    throw;
  }
  CUDA_OK(cudaStreamEndCapture(stream_, &graph));
  const cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  CUDA_OK(e);
  return GraphExec(exec);
}

Executor::Schedule Executor::MakeSchedule(size_t prefix, int cut) {
  Schedule s;
  s.prefix = prefix;
  s.cut = cut;
  if (prefix == 0) return s;
  for (int r : kCuts[cut])
    s.graphs.push_back(Capture([&] {
      for (size_t k = 0; k < prefix; ++k) KERNEL_OK(steps_[k].chunk[r](stream_));
      if (r == kCuts[cut].back()) Enqueue(stream_, prefix);
    }));
  return s;
}

bool Executor::IsDevice(const void* input) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, input) == cudaSuccess) return at.type == cudaMemoryTypeDevice;
  cudaGetLastError();
  return false;
}

// Memory that the copy engine can be given, all of it: a range that is page-locked only in part is not.
bool Executor::IsDirect(const void* p, size_t bytes) {
  auto type_of = [](const void* q) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, q) == cudaSuccess) return at.type;
    cudaGetLastError();
    return cudaMemoryTypeUnregistered;
  };
  const cudaMemoryType first = type_of(p);
  if (first == cudaMemoryTypeHost) return bytes < 2 || type_of((const char*)p + bytes - 1) == cudaMemoryTypeHost;
  return first == cudaMemoryTypeDevice || first == cudaMemoryTypeManaged;
}

// How many leading steps to run part by part, and in which parts: the choice whose inference takes least, timed
// here (best of three each) from page-locked and from pageable memory.  A few counts spread over the range,
// then the neighbours of the best.  (Predicting it from step times and upload rates, as before, missed what
// the launches of a part and the smaller grids cost: SSD-512 batch 8 ran at 712 instead of 661 us.)
void Executor::ChooseSchedules() {
  if (prefix_max_ == 0) return;
  std::vector<char> pageable(in_bytes_, 0);
  auto best_for = [&](const void* input) {
    const Source src = SourceOf(input);
    auto time_of = [&](size_t prefix, int cut) {
      Schedule s = MakeSchedule(prefix, cut);
      double best = 1e30;
      try {
        for (int rep = 0; rep < 4; ++rep) {   // the first is a warm-up
          HostPool::Use helpers;
          if (src == Source::kPool) helpers.Begin(pool());
          const auto t0 = std::chrono::steady_clock::now();
          BeginUpload(input, src);
          Launch(input, src, s, download_ == Download::kPieces ? (char*)heads_[0].host : nullptr, true);
          CUDA_OK(cudaStreamSynchronize(stream_));
          if (down_stream_) CUDA_OK(cudaStreamSynchronize(down_stream_));
          const double t = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
          if (rep > 0) best = std::min(best, t);
        }
      } catch (...) {
        Settle();   // (the input of these timings is about to go)
        throw;
      }
      return best;
    };
    std::map<std::pair<size_t, int>, double> seen;
    auto probe = [&](size_t p, int cut) {
      if (p == 0) cut = 0;
      if (p <= prefix_max_ && !seen.count({p, cut})) seen[{p, cut}] = time_of(p, cut);
    };
    auto best = [&] {
      auto at = seen.begin();
      // (five parts unless others are better by more than a hundredth: the data here are zeros, with
      //  which detection steps take less than they will)
      auto cost = [](const std::pair<const std::pair<size_t, int>, double>& e) { return e.second * (e.first.second ? 1.01 : 1.0); };
      for (auto i = seen.begin(); i != seen.end(); ++i)
        if (cost(*i) < cost(*at)) at = i;
      return at->first;
    };
    if (IsDevice(input)) {   // nothing to wait for: cut only where the head's parts can leave early
      probe(0, 0);
      for (int cut : {0, 1, 2}) probe(prefix_max_, cut);
      return best();
    }
    for (size_t p : {(size_t)0, (size_t)2, (size_t)5, (size_t)9, prefix_max_}) probe(p, 0);
    for (size_t p : {(size_t)2, (size_t)5, (size_t)9, prefix_max_})
      for (int cut : {1, 2}) probe(p, cut);
    for (size_t d : {(size_t)2, (size_t)1}) {
      const auto b = best();
      probe(b.first + d, b.second);
      if (b.first >= d) probe(b.first - d, b.second);
    }
    if (dev_env("CVM_B200_VERBOSE"))
      for (auto& e : seen)
        fprintf(stderr, "%s prefix %zu in %zu parts: %.1f us\n", src == Source::kPool ? "pageable" : "page-locked", e.first.first,
                kCuts[e.first.second].size(), e.second * 1e6);
    return best();
  };
  auto choose = [&](const void* input) {
    const auto b = best_for(input);
    return MakeSchedule(b.first, b.second);
  };
  if (!head_range_end_.empty()) {
    // (an input to time with; where there is no room for it, such inputs go through the whole graph)
    void* dev = nullptr;
    if (cudaMalloc(&dev, in_bytes_) == cudaSuccess) {
      const std::unique_ptr<void, cudaError_t (*)(void*)> hold(dev, cudaFree);
      CUDA_OK(cudaMemset(dev, 0, in_bytes_));
      CUDA_OK(cudaDeviceSynchronize());
      from_device_ = choose(dev);
    } else {
      cudaGetLastError();
    }
  }
  from_pinned_ = choose(in_host_);
  if (in_bytes_ > kSmallInput) from_pageable_ = choose(pageable.data());
}

Executor::~Executor() { Release(); }

void Executor::Release() {
  cudaSetDevice(device_);
  Settle();
  for (Schedule* s : {&from_pinned_, &from_pageable_, &from_device_}) s->graphs.clear();
  graph_whole_.reset();
  graph_staged_.reset();
  kernels_exec_.reset();
  for (auto* events : {&piece_events_, &part_events_, &part_done_})
    for (auto e : *events)
      if (e) cudaEventDestroy(e);
  if (copy_stream_) cudaStreamDestroy(copy_stream_);
  if (down_stream_) cudaStreamDestroy(down_stream_);
  for (void* p : allocs_) cudaFree(p);
  UnmapActivations();
  for (auto& a : act_) vmm().address_free(reinterpret_cast<CUdeviceptr>(a.va), a.va_size);
  for (void* p : pinned_) cudaFreeHost(p);
  if (stream_) cudaStreamDestroy(stream_);
  cudaGetLastError();
}

// Where the bytes of an input come from.  Page-locked (or device) memory is read where it lies.  A
// pageable input of up to 1 MiB is copied into the staging buffer by the calling thread (waking
// helpers costs more than they save: 1 MiB takes about 50 us cold), a larger one by the pool.  A
// page-locked input of up to 256 KiB is staged as well: the copy takes 4 us, and the inference
// is then one graph that begins by fetching the staging buffer.
Executor::Source Executor::SourceOf(const void* input) const {
  if (IsDirect(input, in_bytes_)) return in_bytes_ <= kSmallDirect && graph_staged_ && !IsDevice(input) ? Source::kSmall : Source::kDirect;
  return in_bytes_ <= kSmallInput ? Source::kSmall : Source::kPool;
}

HostPool& Executor::pool() {
  if (!pool_) {
    unsigned hw = std::thread::hardware_concurrency();
    int gpus = 1;
    cudaGetDeviceCount(&gpus);
    // five helpers beside the calling thread, fewer when the host has few cores per GPU: one core
    // copies 14 GB/s here, four just reach the link's 55 GB/s, six leave room for a fill beside it
    pool_.reset(new HostPool(device_, hw ? std::max(1, std::min(5, (int)hw / std::max(1, gpus) - 1)) : 1));
  }
  return *pool_;
}

// After an error: waits for what is queued, so that no copy engine or kernel reads or writes the caller's
// buffers (or the staging buffers of the next call) once the error has been reported.
void Executor::Settle() {
  for (cudaStream_t s : {copy_stream_, stream_, down_stream_})
    if (s) cudaStreamSynchronize(s);
  cudaGetLastError();
  queued_pieces_ = arrived_pieces_ = deliver_units_ = 0;
}

void Executor::BeginUpload(const void* input, Source src) {
  if (src != Source::kPool) return;
  const char* from = (const char*)input;
  char* to = (char*)in_host_;
  const size_t bytes = in_bytes_, pieces = (bytes + kStagePiece - 1) / kStagePiece;
  pool().Start(HostPool::kUpload, pieces, pieces, [from, to, bytes](size_t k) {
    const size_t off = k * kStagePiece;
    stream_copy(to + off, from + off, std::min(kStagePiece, bytes - off));
  });
}

// Staged bytes are sent in groups of pieces (1 MiB) as soon as they are there: fewer driver calls,
// still well pipelined.
void Executor::SendRange(const void* input, Source src, size_t begin, size_t bytes, cudaStream_t s) {
  char* const dev = (char*)in_dev_;
  if (src == Source::kDirect) {
    CUDA_OK(cudaMemcpyAsync(dev + begin, (const char*)input + begin, bytes, cudaMemcpyDefault, s));
    return;
  }
  const size_t group = src == Source::kSmall ? kStagePiece : 4 * kStagePiece;
  for (size_t off = begin; off < begin + bytes;) {
    const size_t end = std::min(begin + bytes, (off / group + 1) * group);
    if (src == Source::kSmall) memcpy((char*)in_host_ + off, (const char*)input + off, end - off);
    else
      for (size_t k = off / kStagePiece; k * kStagePiece < end; ++k) pool().WaitPiece(HostPool::kUpload, k);
    CUDA_OK(cudaMemcpyAsync(dev + off, (char*)in_host_ + off, end - off, cudaMemcpyHostToDevice, s));
    off = end;
    PollPieces();
  }
}

void Executor::Upload(const void* input, cudaStream_t s) {
  const Source src = SourceOf(input);
  HostPool::Use helpers;
  if (src == Source::kPool) helpers.Begin(pool());
  BeginUpload(input, src);
  SendRange(input, src, 0, in_bytes_, s);
}

// Heads of up to 1 MiB in all (256 KiB when they go out as they are: one thread's copy of the rest would
// take longer than its download in pieces; 8 MiB of an NMS head's rows: fetching its -1 tail too costs more) are
// written into page-locked memory by one kernel, with the status word: a copy node for each costs 3 us and more
// and starts only after the kernel before it has drained.  A single larger head whose bytes are
// the result leaves in pieces (DeliverPieces).
void Executor::ChooseDownload() {
  size_t total = 0;
  for (const auto& h : heads_) total += h.live_bytes ? h.images * h.live_bytes : h.bytes;
  const size_t small = plain_ ? (heads_[0].live_bytes ? (size_t)8 << 20 : (size_t)256 << 10) : (size_t)1 << 20;
  if (total <= small && heads_.size() + 2 <= CVMK_MAX_EXPORT_SEGMENTS) {
    download_ = Download::kKernel;
  } else {
    for (auto& h : heads_) h.live_bytes = 0;
    download_ = plain_ ? Download::kPieces : Download::kCopies;
  }
  if (download_ == Download::kPieces) {
    download_piece_ = heads_[0].bytes <= 4 * kDownloadPiece ? kDownloadPiece / 4 : kDownloadPiece;
    if (prefix_max_ != steps_.size()) head_range_end_.clear();
    std::vector<size_t> ends = head_range_end_;   // (no piece crosses the end of a part)
    ends.push_back(heads_[0].bytes);
    std::sort(ends.begin(), ends.end());
    size_t at = 0;
    for (size_t end : ends)
      for (; at < end; at = piece_end_.back()) piece_end_.push_back(std::min(end, at + download_piece_));
    piece_events_.resize(piece_end_.size());
    for (auto& e : piece_events_) CUDA_OK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  }
  if (download_ != Download::kPieces) head_range_end_.clear();
  if (download_ == Download::kKernel && heads_[0].live_bytes) {
    CUDA_OK(cudaMallocHost((void**)&valid_host_, heads_[0].images * 4));
    pinned_.push_back(valid_host_);
  }
}

void Executor::Enqueue(cudaStream_t s, size_t first) {
  for (size_t k = first; k < steps_.size(); ++k) {
    auto& st = steps_[k];
    int rc = st.launch(s);
    CHECK(rc == CVMK_OK) << "step " << st.label << " failed (" << rc << "): " << cvmk_last_error();
  }
  cvmk_export_segment seg[CVMK_MAX_EXPORT_SEGMENTS];
  int n = 0;
  auto add = [&](const void* src, void* dst, size_t rows, size_t row_bytes, size_t pitch) {
    seg[n].src = src; seg[n].dst = dst;
    seg[n].rows = (int64_t)rows; seg[n].row_bytes = (int64_t)row_bytes; seg[n].src_pitch = (int64_t)pitch;
    ++n;
  };
  add(status_dev_, status_host_, 1, 4, 4);
  if (download_ == Download::kKernel) {
    for (auto& h : heads_) {
      if (h.live_bytes) add(h.dev, h.host, h.images, h.live_bytes, h.bytes / h.images);
      else add(h.dev, h.host, 1, h.bytes, h.bytes);
      if (h.live_bytes) add(h.valid_count, valid_host_, 1, h.images * 4, h.images * 4);
    }
  } else if (download_ == Download::kCopies) {
    for (auto& h : heads_) CUDA_OK(cudaMemcpyAsync(h.host, h.dev, h.bytes, cudaMemcpyDeviceToHost, s));
  }
  KERNEL_OK(cvmk_export(seg, n, s));
  if (download_ == Download::kKernel) KERNEL_OK(cvmk_signal(done_host_, s));
}

// Waits for the word that the last kernel writes after the heads: the host sees it some microseconds
// before the stream reports its end.  The stream is asked now and then, so that an error ends the wait.
void Executor::AwaitDone() {
  volatile int32_t* done = done_host_;
  for (uint32_t k = 1; *done == 0; ++k) {
    if ((k & 1023) == 0) {
      const cudaError_t e = cudaStreamQuery(stream_);
      if (e == cudaErrorNotReady) continue;
      CUDA_OK(e);
      break;
    }
    HostPool::Relax();
  }
  std::atomic_thread_fence(std::memory_order_acquire);
}

// The part of an NMS head that is -1 whatever the data says, written while the GPU works.
void Executor::StartFill(char* out) {
  const HeadOut& h = heads_[0];
  const size_t image = h.bytes / h.images, tail = image - h.live_bytes, live = h.live_bytes;
  const size_t per = std::max<size_t>(1, (tail + kStagePiece - 1) / kStagePiece);
  const size_t piece = (tail + per - 1) / per;
  pool().Start(HostPool::kFill, h.images * per, h.images * per, [=](size_t k) {
    const size_t b = k / per, off = std::min(tail, (k % per) * piece);
    stream_fill(out + b * image + live + off, 0xff, std::min(piece, tail - off));
  });
}

// One large head: the copy engine brings it in pieces, the pool copies every piece that has arrived
// into the caller's buffer.  A page-locked buffer takes the pieces directly.
void Executor::StartDelivery(char* out) {
  queued_pieces_ = arrived_pieces_ = 0;
  deliver_units_ = 0;
  if (IsDirect(out, heads_[0].bytes)) return;
  const size_t unit = DeliverUnit(), bytes = heads_[0].bytes;
  const char* from = (const char*)heads_[0].host;
  deliver_units_ = (bytes + unit - 1) / unit;
  pool().Start(HostPool::kDownload, deliver_units_, 0, [=](size_t k) { memcpy(out + k * unit, from + k * unit, std::min(unit, bytes - k * unit)); });
}

// Queues the pieces of the head's first `bytes` that are not queued yet.
void Executor::QueuePieces(char* head, size_t bytes, cudaStream_t s) {
  for (; queued_pieces_ < piece_end_.size() && piece_end_[queued_pieces_] <= bytes; ++queued_pieces_) {
    const size_t at = queued_pieces_ ? piece_end_[queued_pieces_ - 1] : 0;
    CUDA_OK(cudaMemcpyAsync(head + at, (const char*)heads_[0].dev + at, piece_end_[queued_pieces_] - at, cudaMemcpyDefault, s));
    CUDA_OK(cudaEventRecord(piece_events_[queued_pieces_], s));
  }
}

// Hands the pieces that have arrived to the pool.
void Executor::PollPieces() {
  if (!deliver_units_) return;
  const size_t before = arrived_pieces_;
  for (; arrived_pieces_ < queued_pieces_; ++arrived_pieces_) {
    const cudaError_t e = cudaEventQuery(piece_events_[arrived_pieces_]);
    if (e == cudaErrorNotReady) break;
    CUDA_OK(e);
  }
  if (arrived_pieces_ == before) return;
  const bool all = arrived_pieces_ == piece_end_.size();
  pool().Release(HostPool::kDownload, all ? deliver_units_ : piece_end_[arrived_pieces_ - 1] / DeliverUnit());
}

void Executor::DeliverPieces() {
  if (!deliver_units_) {
    CUDA_OK(cudaEventSynchronize(piece_events_.back()));
    return;
  }
  for (PollPieces(); arrived_pieces_ < piece_end_.size(); PollPieces()) pool().HelpOnce();
  pool().Finish(HostPool::kDownload);
  deliver_units_ = 0;
}

// The head is in page-locked memory (and the GPU idle): into the caller's buffer.
void Executor::DeliverHead(char* out, HostPool* awake) {
  const HeadOut& h = heads_[0];
  if (!h.live_bytes) {
    if (!awake || h.bytes < kSmallShare) {
      memcpy(out, h.host, h.bytes);
      return;
    }
    const char* src = (const char*)h.host;
    const size_t bytes = h.bytes, pieces = (bytes + kSmallPiece - 1) / kSmallPiece;
    awake->Start(HostPool::kDownload, pieces, pieces, [=](size_t k) {
      const size_t off = k * kSmallPiece;
      memcpy(out + off, src + off, std::min(kSmallPiece, bytes - off));
    });
    awake->Finish(HostPool::kDownload);
    return;
  }
  const size_t image = h.bytes / h.images, live = h.live_bytes;
  const char* from = (const char*)h.host;
  pool().Start(HostPool::kDownload, h.images, h.images, [=](size_t b) { memcpy(out + b * image, from + b * live, live); });
  pool().Finish(HostPool::kDownload);
  pool().Finish(HostPool::kFill);
  // The operator's loop ends at the first image without valid boxes; what it leaves in the images
  // after that one is whatever their memory holds, which is fetched as it is.
  size_t b = 0;
  while (b < h.images && valid_host_[b] > 0) ++b;
  if (b + 1 < h.images) {
    const size_t at = (b + 1) * image;
    CUDA_OK(cudaMemcpyAsync((char*)h.host + at, (const char*)h.dev + at, h.bytes - at, cudaMemcpyDeviceToHost, stream_));
    CUDA_OK(cudaStreamSynchronize(stream_));
    memcpy(out + at, (const char*)h.host + at, h.bytes - at);
  }
}

// Queues the upload and the kernels of one inference, and the download of its head to `head` when that
// leaves in pieces (null otherwise).  When all of the graph runs part by part, the head's part follows each on a
// stream of its own: both directions of the link and the kernels then work at the same time (64 images of
// 64 -> 64 channels at 56 x 56, 12.8 MB each way: 607 -> 465 us from page-locked memory, 374 -> 346 from the
// device's own).  Without `early` the head leaves after all of the input has been read.
void Executor::Launch(const void* input, Source src, const Schedule& how, char* head, bool early) {
  queued_pieces_ = arrived_pieces_ = 0;
  if (how.prefix == 0) {
    SendRange(input, src, 0, in_bytes_, stream_);
    if (graph_whole_) CUDA_OK(cudaGraphLaunch(graph_whole_.get(), stream_));
    else Enqueue(stream_);
    if (head) QueuePieces(head, heads_[0].bytes, stream_);
    return;
  }
  const bool parts_leave = early && head && how.prefix == steps_.size() && !head_range_end_.empty();
  size_t begin = 0;
  for (size_t c = 0; c < how.graphs.size(); ++c) {
    const int r = kCuts[how.cut][c];
    SendRange(input, src, begin, range_end_[r] - begin, copy_stream_);
    CUDA_OK(cudaEventRecord(part_events_[c], copy_stream_));
    CUDA_OK(cudaStreamWaitEvent(stream_, part_events_[c], 0));
    CUDA_OK(cudaGraphLaunch(how.graphs[c].get(), stream_));
    if (parts_leave) {
      CUDA_OK(cudaEventRecord(part_done_[c], stream_));
      CUDA_OK(cudaStreamWaitEvent(down_stream_, part_done_[c], 0));
      QueuePieces(head, head_range_end_[r], down_stream_);
      PollPieces();
    }
    begin = range_end_[r];
  }
  if (head && !parts_leave) QueuePieces(head, heads_[0].bytes, stream_);
}

void Executor::Run(const void* input, size_t input_bytes, char* out) {
  CHECK(input_bytes == in_bytes_) << "input size " << input_bytes << " vs. " << in_bytes_;
  CUDA_OK(cudaSetDevice(device_));
  try {
    RunOnce(input, out);
  } catch (...) {
    Settle();
    throw;
  }
}

void Executor::RunOnce(const void* input, char* out) {
  const auto called = std::chrono::steady_clock::now();
  const Source src = SourceOf(input);
  const bool on_device = src == Source::kDirect && IsDevice(input);
  const bool fill = plain_ && heads_[0].live_bytes > 0, pieces = plain_ && download_ == Download::kPieces;
  HostPool::Use guard;
  if (src == Source::kPool || fill || pieces) guard.Begin(pool());
  const bool signal = download_ == Download::kKernel;
  if (signal) *(volatile int32_t*)done_host_ = 0;
  BeginUpload(input, src);
  // a caller may have its result where its input is: then nothing is written before all of that is read
  const uintptr_t in_at = (uintptr_t)input, out_at = (uintptr_t)out;
  const bool apart = in_at + in_bytes_ <= out_at || (plain_ && out_at + heads_[0].bytes <= in_at);
  if (fill && apart) StartFill(out);
  if (pieces) StartDelivery(out);
  char* const head = !pieces ? nullptr : (deliver_units_ ? (char*)heads_[0].host : out);   // where the copy engine writes
  if (src == Source::kSmall && graph_staged_) {
    const bool share = in_bytes_ >= kSmallShare;
    if (share && pool_ && pool_->awake()) {
      guard.Begin(*pool_);
      const char* from = (const char*)input;
      char* to = (char*)in_host_;
      const size_t bytes = in_bytes_, pieces = (bytes + kSmallPiece - 1) / kSmallPiece;
      guard.p->Start(HostPool::kUpload, pieces, pieces, [from, to, bytes](size_t k) {
        const size_t off = k * kSmallPiece;
        memcpy(to + off, from + off, std::min(kSmallPiece, bytes - off));
      });
      guard.p->Finish(HostPool::kUpload);
    } else {
      memcpy(in_host_, input, in_bytes_);
    }
    CUDA_OK(cudaGraphLaunch(graph_staged_.get(), stream_));
    if (head) QueuePieces(head, heads_[0].bytes, stream_);
  } else {
    Launch(input, src, on_device ? from_device_ : (src == Source::kDirect ? from_pinned_ : from_pageable_), head, apart);
  }
  // calls that follow one another closely: the helpers wake up while the GPU works, for the head and for
  // the next call's input
  const bool worth = (src == Source::kSmall && in_bytes_ >= kSmallShare) || (signal && plain_ && heads_[0].bytes >= kSmallShare);
  if (worth && !guard.p && called - last_call_ < std::chrono::microseconds(HostPool::kLingerUs)) guard.Begin(pool());
  if (pieces) DeliverPieces();
  else if (signal) AwaitDone();
  else CUDA_OK(cudaStreamSynchronize(stream_));
  if (*status_host_ != 0) {
    const int code = *status_host_;
    *status_host_ = 0;
    cudaMemsetAsync(status_dev_, 0, 4, stream_);
    cudaStreamSynchronize(stream_);
    FATAL() << "a device-side wait ran out (status word 0x" << std::hex << code << ")";
  }
  if (fill && !apart) StartFill(out);
  if (plain_ && !pieces) DeliverHead(out, guard.p);
  last_call_ = std::chrono::steady_clock::now();
}

std::string Executor::DescribeSchedules() const {
  std::ostringstream os;
  const std::pair<const char*, const Schedule*> all[] = {{"pinned", &from_pinned_}, {"pageable", &from_pageable_}, {"device", &from_device_}};
  for (const auto& s : all) os << s.first << "\t" << s.second->prefix << "\t" << std::max<size_t>(1, s.second->graphs.size()) << "\n";
  return os.str();
}

void Executor::SetStatusWord(int code) {
  CUDA_OK(cudaSetDevice(device_));
  const int32_t v = code;
  CUDA_OK(cudaMemcpyAsync(status_dev_, &v, sizeof(v), cudaMemcpyHostToDevice, stream_));
  CUDA_OK(cudaStreamSynchronize(stream_));
}

namespace {
class TimingEvents {
 public:
  explicit TimingEvents(size_t n) {
    for (size_t k = 0; k < n; ++k) {
      cudaEvent_t e = nullptr;
      CUDA_OK(cudaEventCreate(&e));
      e_.emplace_back(e, cudaEventDestroy);
    }
  }
  cudaEvent_t operator[](size_t k) const { return e_[k].get(); }

 private:
  std::vector<std::unique_ptr<CUevent_st, cudaError_t (*)(cudaEvent_t)>> e_;
};
}  // namespace

float Executor::ReplayDevice(int iters) {
  CHECK(iters > 0);
  CUDA_OK(cudaSetDevice(device_));
  if (use_graph_ && !kernels_exec_)
    kernels_exec_ = Capture([this] {
      for (auto& st : steps_) KERNEL_OK(st.launch(stream_));
    });
  TimingEvents ev(2);
  CUDA_OK(cudaEventRecord(ev[0], stream_));
  for (int i = 0; i < iters; ++i) {
    if (kernels_exec_) CUDA_OK(cudaGraphLaunch(kernels_exec_.get(), stream_));
    else for (auto& st : steps_) KERNEL_OK(st.launch(stream_));
  }
  CUDA_OK(cudaEventRecord(ev[1], stream_));
  CUDA_OK(cudaEventSynchronize(ev[1]));
  float ms = 0;
  CUDA_OK(cudaEventElapsedTime(&ms, ev[0], ev[1]));
  return ms;
}

std::vector<std::pair<std::string, float>> Executor::ProfileOnce(const void* input, size_t input_bytes) {
  CHECK(input_bytes == in_bytes_);
  CUDA_OK(cudaSetDevice(device_));
  std::vector<std::pair<std::string, float>> out;
  TimingEvents ev(steps_.size() + 1);
  try {
    Upload(input, stream_);
    CUDA_OK(cudaEventRecord(ev[0], stream_));
    for (size_t i = 0; i < steps_.size(); ++i) {
      KERNEL_OK(steps_[i].launch(stream_));
      CUDA_OK(cudaEventRecord(ev[i + 1], stream_));
    }
    CUDA_OK(cudaStreamSynchronize(stream_));
  } catch (...) {
    Settle();
    throw;
  }
  for (size_t i = 0; i < steps_.size(); ++i) {
    float ms = 0;
    CUDA_OK(cudaEventElapsedTime(&ms, ev[i], ev[i + 1]));
    out.emplace_back(steps_[i].label, ms);
  }
  return out;
}

}  // namespace cvm
