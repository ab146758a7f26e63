// Python module `quant_cuda`: same name, function names, argument order and dtypes as
// the reference's extension (csrc/quant_cuda.cpp:41-77 of the reference project), so
// that llama/qlinear.py and benchmark_speed.py of the reference run against it
// unchanged.  This file holds no device code: it validates the tensors, picks the
// current CUDA stream and device, and calls the C ABI declared in include/cherryq.h.
// Differences from the reference, all deliberate:
//   * work is enqueued on torch's CURRENT stream (the reference uses the legacy
//     default stream), so the ops can be captured in CUDA graphs;
//   * a device guard covers all four ops (the reference guards only the matmuls);
//   * wrong dtypes / devices / shapes / group sizes raise RuntimeError (the
//     reference's 3-bit op silently does nothing for an unsupported group size).
// The first matmul call with a given set of weight tensors re-packs them on the GPU
// (allocates and synchronises), so it must happen before any stream capture.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/core/InferenceMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>
#include <cmath>

#include <array>
#include <map>
#include <mutex>
#include <vector>

#include "cherryq.h"

namespace {

void check_status(int rc, const char* what) {
  if (rc == CQ_OK) return;
  if (rc == CQ_ERR_CUDA) {
    TORCH_CHECK(false, what, ": CUDA error ", cq_last_cuda_error());
  }
  TORCH_CHECK(false, what, ": ", cq_strerror(rc));
}

void check_tensor(const torch::Tensor& t, const char* name, c10::ScalarType dtype, const torch::Tensor& like) {
  TORCH_CHECK(t.defined(), name, " is undefined");
  TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
  TORCH_CHECK(t.scalar_type() == dtype, name, " must have dtype ", c10::toString(dtype), ", got ",
              c10::toString(t.scalar_type()));
  TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
  TORCH_CHECK(t.device() == like.device(), name, " is on ", t.device(), " but vec is on ", like.device());
}

cq_stream_t current_stream() { return (cq_stream_t)c10::cuda::getCurrentCUDAStream().stream(); }

// The C library caches re-packed copies by buffer ADDRESS.  Torch's allocator hands a freed block to
// the next tensor of the same size, so an address alone does not identify a buffer: every cached set
// is paired here with weak references to the four tensors' storages.  A call whose storages are not
// the ones on record (or whose record has expired) evicts the library's copies for these addresses
// before it proceeds, and every such miss also sweeps the records whose storages have died, which
// frees their copies.  The reference's ops keep no state at all (csrc/quant_cuda.cpp:56-69).
struct StorageGuard {
  std::vector<c10::weak_intrusive_ptr<c10::StorageImpl>> w;   // four entries
  const void* ptr[4];
  int device;
};
std::mutex g_guard_mu;
std::map<std::array<const void*, 4>, StorageGuard> g_guards;

void guard_buffers(const torch::Tensor& q, const torch::Tensor& s, const torch::Tensor& cw, const torch::Tensor& ci) {
  const torch::Tensor* t[4] = {&q, &s, &cw, &ci};
  std::array<const void*, 4> key = {q.data_ptr(), s.data_ptr(), cw.data_ptr(), ci.data_ptr()};
  std::lock_guard<std::mutex> lock(g_guard_mu);
  auto it = g_guards.find(key);
  if (it != g_guards.end()) {
    bool same = true;
    for (int i = 0; i < 4; ++i) {
      auto sp = it->second.w[i].lock();
      same = same && sp && sp.get() == t[i]->storage().unsafeGetStorageImpl();
    }
    if (same) return;
    g_guards.erase(it);
  }
  // unknown or recycled addresses: whatever the library holds for them is stale
  cq_cache_evict(key[0], key[1], key[2], key[3]);
  for (auto g = g_guards.begin(); g != g_guards.end();) {
    bool dead = false;
    for (int i = 0; i < 4; ++i) dead = dead || g->second.w[i].expired();
    if (dead) {
      const at::cuda::OptionalCUDAGuard dg(c10::Device(c10::kCUDA, (c10::DeviceIndex)g->second.device));
      cq_cache_evict(g->second.ptr[0], g->second.ptr[1], g->second.ptr[2], g->second.ptr[3]);
      g = g_guards.erase(g);
    } else {
      ++g;
    }
  }
  StorageGuard ng;
  for (int i = 0; i < 4; ++i) {
    ng.w.push_back(t[i]->storage().getWeakStorageImpl());
    ng.ptr[i] = key[i];
  }
  ng.device = q.device().index();
  g_guards.emplace(key, std::move(ng));
}

uint64_t version_tag(const torch::Tensor& a, const torch::Tensor& b, const torch::Tensor& c,
                     const torch::Tensor& d) {
  // inference tensors (created under torch.inference_mode) keep no version counter
  auto v = [](const torch::Tensor& t) -> uint64_t { return t.is_inference() ? 0u : (uint64_t)t._version(); };
  return v(a) + (v(b) << 16) + (v(c) << 32) + (v(d) << 48);
}

void vecquant3matmul_cherryq(torch::Tensor vec, torch::Tensor qweight, torch::Tensor cherry_weight,
                             torch::Tensor cherry_indices, torch::Tensor scaling_factors, torch::Tensor mul,
                             int group_size, bool fp16) {
  const at::cuda::OptionalCUDAGuard device_guard(device_of(vec));
  const auto ft = fp16 ? torch::kFloat16 : torch::kFloat32;
  const auto it = fp16 ? torch::kInt16 : torch::kInt32;
  check_tensor(vec, "vec", ft, vec);
  check_tensor(qweight, "qweight", torch::kUInt8, vec);
  check_tensor(cherry_weight, "cherry_weight", ft, vec);
  check_tensor(cherry_indices, "cherry_indices", it, vec);
  check_tensor(scaling_factors, "scaling_factors", ft, vec);
  check_tensor(mul, "mul", ft, vec);
  TORCH_CHECK(vec.dim() == 2 && qweight.dim() == 2 && mul.dim() == 2, "vec, qweight and mul must be 2-D");
  TORCH_CHECK(mul.size(0) == vec.size(0) && mul.size(1) == qweight.size(1), "mul must be (batch, width)");
  TORCH_CHECK(cherry_weight.numel() == cherry_indices.size(0) * qweight.size(1), "cherry_weight must be (C, width)");
  if (fp16) guard_buffers(qweight, scaling_factors, cherry_weight, cherry_indices);
  check_status(cq_vecquant3matmul_cherryq(
                   vec.data_ptr(), qweight.data_ptr<uint8_t>(), cherry_weight.data_ptr(), cherry_indices.data_ptr(),
                   scaling_factors.data_ptr(), mul.data_ptr(), (int)vec.size(0), (int)vec.size(1),
                   (int)qweight.size(0), (int)qweight.size(1), (int)cherry_indices.size(0), group_size, fp16 ? 1 : 0,
                   version_tag(qweight, cherry_weight, cherry_indices, scaling_factors), current_stream()),
               "vecquant3matmul_cherryq");
}

void vecquant4matmul_cherryq(torch::Tensor vec, torch::Tensor qweight, torch::Tensor cherry_weight,
                             torch::Tensor cherry_indices, torch::Tensor scaling_factors, torch::Tensor mul,
                             int group_size) {
  const at::cuda::OptionalCUDAGuard device_guard(device_of(vec));
  check_tensor(vec, "vec", torch::kFloat16, vec);
  check_tensor(qweight, "qweight", torch::kUInt8, vec);
  check_tensor(cherry_weight, "cherry_weight", torch::kFloat16, vec);
  check_tensor(cherry_indices, "cherry_indices", torch::kInt16, vec);
  check_tensor(scaling_factors, "scaling_factors", torch::kFloat16, vec);
  check_tensor(mul, "mul", torch::kFloat16, vec);
  TORCH_CHECK(vec.dim() == 2 && qweight.dim() == 2 && mul.dim() == 2, "vec, qweight and mul must be 2-D");
  TORCH_CHECK(mul.size(0) == vec.size(0) && mul.size(1) == qweight.size(1), "mul must be (batch, width)");
  TORCH_CHECK(cherry_weight.numel() == cherry_indices.size(0) * qweight.size(1), "cherry_weight must be (C, width)");
  guard_buffers(qweight, scaling_factors, cherry_weight, cherry_indices);
  check_status(cq_vecquant4matmul_cherryq(
                   vec.data_ptr(), qweight.data_ptr<uint8_t>(), cherry_weight.data_ptr(),
                   (const int16_t*)cherry_indices.data_ptr(), scaling_factors.data_ptr(), mul.data_ptr(),
                   (int)vec.size(0), (int)vec.size(1), (int)qweight.size(0), (int)qweight.size(1),
                   (int)cherry_indices.size(0), group_size,
                   version_tag(qweight, cherry_weight, cherry_indices, scaling_factors), current_stream()),
               "vecquant4matmul_cherryq");
}

void dequantize_normal(int bits, torch::Tensor qweight, torch::Tensor scaling_factors, torch::Tensor out, int height,
                       int cherry_size, int group_size) {
  const at::cuda::OptionalCUDAGuard device_guard(device_of(qweight));
  check_tensor(qweight, "qweight", torch::kUInt8, qweight);
  check_tensor(scaling_factors, "scaling_factors", torch::kFloat32, qweight);
  check_tensor(out, "out", torch::kFloat32, qweight);
  TORCH_CHECK(qweight.dim() == 2 && out.dim() == 2 && out.size(1) == qweight.size(1) &&
                  out.size(0) >= height - cherry_size,
              "out must be (>= height - cherry_size, width)");
  auto fn = bits == 3 ? cq_dequantize3_normal : cq_dequantize4_normal;
  check_status(fn(qweight.data_ptr<uint8_t>(), scaling_factors.data_ptr<float>(), out.data_ptr<float>(),
                  (int)qweight.size(0), (int)qweight.size(1), height, cherry_size, group_size, current_stream()),
               bits == 3 ? "Dequantize3Normal" : "Dequantize4Normal");
}

void Dequantize3Normal(torch::Tensor qweight, torch::Tensor scaling_factors, torch::Tensor out, int height,
                       int cherry_size, int group_size) {
  dequantize_normal(3, qweight, scaling_factors, out, height, cherry_size, group_size);
}
void Dequantize4Normal(torch::Tensor qweight, torch::Tensor scaling_factors, torch::Tensor out, int height,
                       int cherry_size, int group_size) {
  dequantize_normal(4, qweight, scaling_factors, out, height, cherry_size, group_size);
}

// ------------------------------------------------------------------ additive entry points
// GPU QuantLinear.pack (llama/qlinear.py:67-118): returns (qweight, scales, cherry_weight, cherry_indices).
std::vector<torch::Tensor> pack(torch::Tensor weight, torch::Tensor cherry_unsorted, int bits, int group_size) {
  const at::cuda::OptionalCUDAGuard device_guard(device_of(weight));
  TORCH_CHECK(weight.is_cuda() && weight.dim() == 2 && weight.is_contiguous(), "weight must be a contiguous 2-D CUDA tensor");
  TORCH_CHECK(weight.scalar_type() == torch::kFloat16 || weight.scalar_type() == torch::kFloat32,
              "weight must be float16 or float32");
  check_tensor(cherry_unsorted, "cherry_indices", torch::kInt32, weight);
  const int N = (int)weight.size(0), K = (int)weight.size(1), C = (int)cherry_unsorted.numel();
  const int G = group_size == -1 ? K : group_size;
  TORCH_CHECK(G > 0, "group_size must be positive or -1");
  TORCH_CHECK(K % 8 == 0 && N % 8 == 0 && C % 8 == 0 && C < K, "in_features, out_features and the cherry count must be multiples of 8");
  auto u8 = torch::TensorOptions().device(weight.device()).dtype(torch::kUInt8);
  auto qweight = torch::empty({(K - C) / 8 * bits, N}, u8);
  auto scales = torch::empty({(K - C + G - 1) / G, N}, u8.dtype(torch::kFloat16));
  auto cw = torch::empty({C, N}, u8.dtype(torch::kFloat16));
  auto idx = torch::empty({C}, u8.dtype(torch::kInt16));
  check_status(cq_pack(weight.data_ptr(), weight.scalar_type() == torch::kFloat32, cherry_unsorted.data_ptr<int32_t>(),
                       bits, K, N, C, G, qweight.data_ptr<uint8_t>(), scales.data_ptr(), cw.data_ptr(),
                       (int16_t*)idx.data_ptr(), nullptr, current_stream()),
               "pack");
  return {qweight, scales, cw, idx};
}

// Fake-quantised training weight (llama/cherry_linear.py:69-99); `quantised` marks the columns that are not cherries.
torch::Tensor fake_quant(torch::Tensor weight, torch::Tensor quantised, int bits, int group_size, bool ste) {
  const at::cuda::OptionalCUDAGuard device_guard(device_of(weight));
  TORCH_CHECK(weight.is_cuda() && weight.dim() == 2 && weight.is_contiguous(), "weight must be a contiguous 2-D CUDA tensor");
  const auto t = weight.scalar_type();
  TORCH_CHECK(t == torch::kFloat16 || t == torch::kFloat32 || t == torch::kBFloat16, "weight must be float16, float32 or bfloat16");
  check_tensor(quantised, "quantised", torch::kBool, weight);
  TORCH_CHECK(quantised.numel() == weight.size(1), "quantised must have one entry per column");
  auto out = torch::empty_like(weight);
  auto table = torch::empty({weight.size(1) / 8}, weight.options().dtype(torch::kInt32));
  check_status(cq_fake_quant(weight.data_ptr(), t == torch::kFloat16 ? 0 : (t == torch::kFloat32 ? 1 : 2),
                             (const uint8_t*)quantised.data_ptr(), bits, (int)weight.size(1), (int)weight.size(0), group_size,
                             ste ? 1 : 0, out.data_ptr(), (uint32_t*)table.data_ptr(), current_stream()),
               "fake_quant");
  return out;
}

// GPU QuantLinear.unpack (llama/qlinear.py:120-162): dense (N, K) fp16.
torch::Tensor unpack_dense(torch::Tensor qweight, torch::Tensor scales, torch::Tensor cherry_weight,
                           torch::Tensor cherry_indices, int bits, int in_features, int group_size) {
  const at::cuda::OptionalCUDAGuard device_guard(device_of(qweight));
  check_tensor(qweight, "qweight", torch::kUInt8, qweight);
  check_tensor(scales, "scales", torch::kFloat16, qweight);
  check_tensor(cherry_weight, "cherry_weight", torch::kFloat16, qweight);
  check_tensor(cherry_indices, "cherry_indices", torch::kInt16, qweight);
  const int N = (int)qweight.size(1), C = (int)cherry_indices.numel();
  auto dense = torch::empty({N, in_features}, scales.options());
  check_status(cq_unpack_dense(qweight.data_ptr<uint8_t>(), scales.data_ptr(), cherry_weight.data_ptr(),
                               (const int16_t*)cherry_indices.data_ptr(), bits, in_features, N, C, group_size,
                               dense.data_ptr(), current_stream()),
               "unpack_dense");
  return dense;
}

std::mutex g_mu;
std::map<int, torch::Tensor> g_scratch;  // per device: matvec scratch followed by a status word

// Workspace of the decode attention, per device, grow-only.  The counters of every call end at `counters` bytes, where the
// partial results begin: calls of different numbers of heads share the buffer and none writes over the zeros that another
// counts from.  Outgrown buffers are kept, since a captured graph may hold their addresses; sizes at least double.
struct AttnWorkspace {
  torch::Tensor now;
  size_t counters = 0;
  std::vector<torch::Tensor> outgrown;
};
std::map<int, AttnWorkspace> g_attn_ws;

// the workspace of a call of `heads` heads (in all sequences) that needs `bytes`; `keep` holds the buffer
void* attn_workspace(const torch::Device& dev, size_t heads, size_t bytes, torch::Tensor* keep) {
  const size_t own = (heads * sizeof(unsigned int) + 255) / 256 * 256;
  const auto options = torch::TensorOptions().device(dev).dtype(torch::kUInt8);
  std::lock_guard<std::mutex> lock(g_mu);
  auto& w = g_attn_ws[dev.index()];
  if (w.counters < own || !w.now.defined() || (size_t)w.now.numel() < w.counters + bytes) {
    // a buffer made under capture is the graph's own: its zeros are written when the graph runs
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) {
      *keep = torch::zeros({(int64_t)bytes}, options);
      return keep->data_ptr();
    }
    const size_t counters = std::max(own, 2 * w.counters);
    const size_t size = std::max(counters + bytes, w.now.defined() ? 2 * (size_t)w.now.numel() : 0);
    auto t = torch::zeros({(int64_t)size}, options);
    if (w.now.defined()) w.outgrown.push_back(w.now);
    w.now = t;
    w.counters = counters;
  }
  *keep = w.now;
  return w.now.data_ptr<uint8_t>() + w.counters - own;
}

torch::Tensor scratch_for(const torch::Device& dev) {
  std::lock_guard<std::mutex> lock(g_mu);
  auto it = g_scratch.find(dev.index());
  if (it == g_scratch.end()) {
    auto t = torch::zeros({(int64_t)cq_scratch_bytes() + 256}, torch::TensorOptions().device(dev).dtype(torch::kUInt8));
    it = g_scratch.emplace(dev.index(), t).first;
  }
  return it->second;
}

// The device memory of a re-packed layer, and the stream that it was allocated on.  Launches on any stream read it.  Those
// on its own need no record (the allocator gives a freed block out in that stream's order); one on another stream is
// recorded, so that the block is not given out before it ends.
struct LayerBlob {
  torch::Tensor t;
  c10::optional<c10::cuda::CUDAStream> home;

  // A re-pack is finished before the first launch (which reads weights ahead of stream order, or runs on another stream),
  // and a captured one would only run with the graph: neither can happen under capture.
  void allocate(uint64_t bytes, const torch::TensorOptions& options, const char* what) {
    TORCH_CHECK(c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None, what,
                ": the first call of a layer re-packs its weights and cannot be captured; call it once before the capture");
    home = c10::cuda::getCurrentCUDAStream();
    t = torch::empty({(int64_t)bytes}, options);
  }
  void finish() const { home->synchronize(); }
  void use() const {
    const auto now = c10::cuda::getCurrentCUDAStream(t.device().index());
    if (!home || now != *home) c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), now);
  }
};

// The four reference buffers of a layer of which the re-pack kernels read Kc / 8 * bits x N codes, ceil(Kc / G) x N scales
// and C x N cherry weights.
void check_buffers(const torch::Tensor& qweight, const torch::Tensor& scales, const torch::Tensor& cherry_weight,
                   const torch::Tensor& cherry_indices, int bits, int Kc, int G) {
  check_tensor(qweight, "qweight", torch::kUInt8, qweight);
  check_tensor(scales, "scales", torch::kFloat16, qweight);
  check_tensor(cherry_weight, "cherry_weight", torch::kFloat16, qweight);
  check_tensor(cherry_indices, "cherry_indices", torch::kInt16, qweight);
  TORCH_CHECK(qweight.dim() == 2 && qweight.size(0) == Kc / 8 * bits, "qweight must be (", Kc / 8 * bits, ", N)");
  const int64_t N = qweight.size(1);
  TORCH_CHECK(scales.dim() == 2 && scales.size(0) == (Kc + G - 1) / G && scales.size(1) == N, "scales must be (ceil(K'/G), N)");
  TORCH_CHECK(cherry_weight.numel() == cherry_indices.numel() * N, "cherry_weight must be (C, N)");
}

// A layer re-packed into the stream layout; owns its device blob.
struct PreparedLayer {
  cq_layer layer;
  LayerBlob blob;

  PreparedLayer(torch::Tensor qweight, torch::Tensor scales, torch::Tensor cherry_weight,
                torch::Tensor cherry_indices, int bits, int in_features, int group_size) {
    const at::cuda::OptionalCUDAGuard device_guard(device_of(qweight));
    TORCH_CHECK(qweight.dim() == 2, "qweight must be 2-D");
    const int N = (int)qweight.size(1), C = (int)cherry_indices.numel();
    check_status(cq_layer_init(&layer, bits, in_features, N, C, group_size, nullptr), "PreparedLayer");
    check_buffers(qweight, scales, cherry_weight, cherry_indices, bits, layer.Kc, layer.G);
    blob.allocate(layer.blob_bytes, qweight.options(), "PreparedLayer");
    layer.blob = blob.t.data_ptr();
    check_status(cq_layer_prepare(&layer, qweight.data_ptr<uint8_t>(), scales.data_ptr(), cherry_weight.data_ptr(),
                                  (const int16_t*)cherry_indices.data_ptr(), current_stream()),
                 "PreparedLayer");
    blob.finish();
  }

  // A layer rebuilt around an existing blob (e.g. loaded from a file or sliced from a shard).
  PreparedLayer(torch::Tensor blob_, int bits, int in_features, int out_features, int num_cherries, int group_size) {
    TORCH_CHECK(blob_.is_cuda() && blob_.scalar_type() == torch::kUInt8 && blob_.is_contiguous(), "blob must be a contiguous CUDA uint8 tensor");
    check_status(cq_layer_init(&layer, bits, in_features, out_features, num_cherries, group_size, nullptr), "PreparedLayer");
    TORCH_CHECK((uint64_t)blob_.numel() == layer.blob_bytes, "blob has ", blob_.numel(), " bytes, expected ", layer.blob_bytes);
    TORCH_CHECK(((uintptr_t)blob_.data_ptr() & 255) == 0, "blob must be 256-byte aligned");
    blob.t = blob_;
    layer.blob = blob.t.data_ptr();
  }

  // out (M, N) fp16 = [out +] x (M, K) fp16 . W^T
  void matvec(torch::Tensor x, torch::Tensor out, bool accumulate) {
    const at::cuda::OptionalCUDAGuard device_guard(device_of(x));
    check_tensor(x, "x", torch::kFloat16, blob.t);
    check_tensor(out, "out", torch::kFloat16, blob.t);
    TORCH_CHECK(x.dim() == 2 && x.size(1) == layer.K, "x must be (M, ", layer.K, ")");
    TORCH_CHECK(out.dim() == 2 && out.size(0) == x.size(0) && out.size(1) == layer.N, "out must be (M, ", layer.N, ")");
    auto scratch = scratch_for(x.device());
    blob.use();
    uint8_t* sp = scratch.data_ptr<uint8_t>();
    check_status(cq_layer_matvec(&layer, x.data_ptr(), layer.K, out.data_ptr(), layer.N, (int)x.size(0),
                                 accumulate ? 1 : 0, sp, (uint32_t*)(sp + cq_scratch_bytes()), current_stream()),
                 "PreparedLayer.matvec");
  }

  // Back to the reference's four buffers: (qweight, scales, cherry_weight, cherry_indices).
  std::vector<torch::Tensor> unprepare() {
    const at::cuda::OptionalCUDAGuard device_guard(device_of(blob.t));
    auto o = blob.t.options();
    blob.use();
    auto qweight = torch::empty({layer.Kc / 8 * layer.bits, layer.N}, o);
    auto scales = torch::empty({(layer.Kc + layer.G - 1) / layer.G, layer.N}, o.dtype(torch::kFloat16));
    auto cw = torch::empty({layer.C, layer.N}, o.dtype(torch::kFloat16));
    auto idx = torch::empty({layer.C}, o.dtype(torch::kInt16));
    check_status(cq_layer_unprepare(&layer, qweight.data_ptr<uint8_t>(), scales.data_ptr(), cw.data_ptr(),
                                    (int16_t*)idx.data_ptr(), current_stream()),
                 "PreparedLayer.unprepare");
    return {qweight, scales, cw, idx};
  }
};

// A layer re-packed into the row-tile layout of the one-row decode kernel; owns its device blob.
struct RowLayer {
  cq_rlayer layer;
  LayerBlob blob;

  // rows up to which such a layer takes the row kernel on the current device; 0 = the kernel does not take it
  static int row_limit(int bits, int in_features, int out_features, int num_cherries, int group_size) {
    cq_rlayer L;
    if (cq_rlayer_init(&L, bits, in_features, out_features, num_cherries, group_size, nullptr) != CQ_OK) return 0;
    return cq_rlayer_check(&L) == CQ_OK ? cq_rlayer_preferred_rows(&L) : 0;
  }
  static bool supported(int bits, int in_features, int out_features, int num_cherries, int group_size) {
    return row_limit(bits, in_features, out_features, num_cherries, group_size) > 0;
  }

  RowLayer(torch::Tensor qweight, torch::Tensor scales, torch::Tensor cherry_weight, torch::Tensor cherry_indices,
           int bits, int in_features, int group_size) {
    const at::cuda::OptionalCUDAGuard device_guard(device_of(qweight));
    TORCH_CHECK(qweight.dim() == 2, "qweight must be 2-D");
    const int N = (int)qweight.size(1), C = (int)cherry_indices.numel();
    check_status(cq_rlayer_init(&layer, bits, in_features, N, C, group_size, nullptr), "RowLayer");
    check_status(cq_rlayer_check(&layer), "RowLayer");
    check_buffers(qweight, scales, cherry_weight, cherry_indices, bits, layer.Kc, layer.G);
    blob.allocate(layer.blob_bytes, qweight.options(), "RowLayer");
    layer.blob = blob.t.data_ptr();
    check_status(cq_rlayer_prepare(&layer, qweight.data_ptr<uint8_t>(), scales.data_ptr(), cherry_weight.data_ptr(),
                                   (const int16_t*)cherry_indices.data_ptr(), current_stream()),
                 "RowLayer");
    blob.finish();
  }

  // out (M, N) fp16 = [out +] x (M, K) fp16 . W^T; four rows per launch
  void matvec(torch::Tensor x, torch::Tensor out, bool accumulate) {
    const at::cuda::OptionalCUDAGuard device_guard(device_of(x));
    check_tensor(x, "x", torch::kFloat16, blob.t);
    check_tensor(out, "out", torch::kFloat16, blob.t);
    TORCH_CHECK(x.numel() % layer.K == 0 && x.numel() > 0, "x must hold rows of ", layer.K, " activations");
    const int M = (int)(x.numel() / layer.K);
    TORCH_CHECK(out.numel() == (int64_t)M * layer.N, "out must hold ", M, " rows of ", layer.N, " values");
    auto scratch = scratch_for(x.device());
    blob.use();
    uint8_t* sp = scratch.data_ptr<uint8_t>();
    const cq_rlayer* lp = &layer;
    void* yp = out.data_ptr();
    check_status(cq_rlayers_matvec(&lp, 1, x.data_ptr(), layer.K, &yp, layer.N, M, accumulate ? 1 : 0,
                                   (uint32_t*)(sp + cq_scratch_bytes()), current_stream()),
                 "RowLayer.matvec");
  }

  // out (M, N) fp16 = (silu(gate) * up) (M, K) . W^T: the SwiGLU of a gated MLP folded into the down projection
  void matvec_swiglu(torch::Tensor gate, torch::Tensor up, torch::Tensor out) {
    const at::cuda::OptionalCUDAGuard device_guard(device_of(gate));
    check_tensor(gate, "gate", torch::kFloat16, blob.t);
    check_tensor(up, "up", torch::kFloat16, blob.t);
    check_tensor(out, "out", torch::kFloat16, blob.t);
    TORCH_CHECK(gate.sizes() == up.sizes() && gate.numel() % layer.K == 0 && gate.numel() > 0,
                "gate and up must hold the same rows of ", layer.K, " values");
    const int M = (int)(gate.numel() / layer.K);
    TORCH_CHECK(out.numel() == (int64_t)M * layer.N, "out must hold ", M, " rows of ", layer.N, " values");
    auto scratch = scratch_for(gate.device());
    blob.use();
    uint8_t* sp = scratch.data_ptr<uint8_t>();
    check_status(cq_rlayer_matvec_swiglu(&layer, gate.data_ptr(), up.data_ptr(), layer.K, out.data_ptr(), layer.N, M,
                                         (uint32_t*)(sp + cq_scratch_bytes()), current_stream()),
                 "RowLayer.matvec_swiglu");
  }

  // Column-parallel shard: y_local (M, N) = x (M, K) . W^T and, in the same launch, the exchange of the ranks'
  // slices over peer memory: y_all (M, P * N).  regions: the P mapped region addresses (parallel.PeerAllGather).
  void matvec_gather(torch::Tensor x, torch::Tensor y_local, torch::Tensor y_all, std::vector<int64_t> regions, int rank,
                     int64_t capacity, int timeout_ms, torch::Tensor status) {
    const at::cuda::OptionalCUDAGuard device_guard(device_of(x));
    check_tensor(x, "x", torch::kFloat16, blob.t);
    check_tensor(y_local, "y_local", torch::kFloat16, blob.t);
    check_tensor(y_all, "y_all", torch::kFloat16, blob.t);
    check_tensor(status, "status", torch::kInt32, blob.t);
    TORCH_CHECK(x.numel() % layer.K == 0 && x.numel() > 0, "x must hold rows of ", layer.K, " activations");
    const int M = (int)(x.numel() / layer.K), P = (int)regions.size();
    TORCH_CHECK(y_local.numel() == (int64_t)M * layer.N && y_all.numel() == (int64_t)M * layer.N * P,
                "y_local must be (M, N) and y_all (M, P * N)");
    std::vector<void*> rp(P);
    blob.use();
    for (int i = 0; i < P; ++i) rp[i] = (void*)(uintptr_t)regions[i];
    check_status(cq_rlayer_matvec_gather(&layer, x.data_ptr(), layer.K, y_local.data_ptr(), M, rp.data(), P, rank,
                                         (size_t)capacity, y_all.data_ptr(), timeout_ms, (uint32_t*)status.data_ptr(),
                                         current_stream()),
                 "RowLayer.matvec_gather");
  }

  // Back to the reference's four buffers: (qweight, scales, cherry_weight, cherry_indices).
  std::vector<torch::Tensor> unprepare() {
    const at::cuda::OptionalCUDAGuard device_guard(device_of(blob.t));
    auto o = blob.t.options();
    blob.use();
    auto qweight = torch::empty({layer.Kc / 8 * layer.bits, layer.N}, o);
    auto scales = torch::empty({(layer.Kc + layer.G - 1) / layer.G, layer.N}, o.dtype(torch::kFloat16));
    auto cw = torch::empty({layer.C, layer.N}, o.dtype(torch::kFloat16));
    auto idx = torch::empty({layer.C}, o.dtype(torch::kInt16));
    check_status(cq_rlayer_unprepare(&layer, qweight.data_ptr<uint8_t>(), scales.data_ptr(), cw.data_ptr(),
                                     (int16_t*)idx.data_ptr(), current_stream()),
                 "RowLayer.unprepare");
    return {qweight, scales, cw, idx};
  }
};

// A layer re-packed into the tile layout of the tensor-core GEMM (prefill and large batches); owns its blob.
struct TileLayer {
  cq_tlayer layer;
  LayerBlob blob;

  TileLayer(torch::Tensor qweight, torch::Tensor scales, torch::Tensor cherry_weight, torch::Tensor cherry_indices,
            int bits, int in_features, int group_size) {
    const at::cuda::OptionalCUDAGuard device_guard(device_of(qweight));
    TORCH_CHECK(qweight.dim() == 2, "qweight must be 2-D");
    const int N = (int)qweight.size(1), C = (int)cherry_indices.numel();
    check_status(cq_tlayer_init(&layer, bits, in_features, N, C, group_size, nullptr), "TileLayer");
    check_buffers(qweight, scales, cherry_weight, cherry_indices, bits, layer.Kc, layer.G);
    blob.allocate(layer.blob_bytes, qweight.options(), "TileLayer");
    layer.blob = blob.t.data_ptr();
    check_status(cq_tlayer_prepare(&layer, qweight.data_ptr<uint8_t>(), scales.data_ptr(), cherry_weight.data_ptr(),
                                   (const int16_t*)cherry_indices.data_ptr(), current_stream()),
                 "TileLayer");
    blob.finish();
  }

  // out (M, N) fp16 = [out +] x (M, K) fp16 . W^T, walked in slices of 4096 rows (bounds the workspace)
  void gemm(torch::Tensor x, torch::Tensor out, bool accumulate) { gemm_bias(x, out, accumulate, nullptr); }
  // bias: null, or N fp16 values added to the rounded outputs
  void gemm_bias(const torch::Tensor& x, const torch::Tensor& out, bool accumulate, const void* bias) {
    const at::cuda::OptionalCUDAGuard device_guard(device_of(x));
    check_tensor(x, "x", torch::kFloat16, blob.t);
    check_tensor(out, "out", torch::kFloat16, blob.t);
    TORCH_CHECK(x.dim() == 2 && x.size(1) == layer.K, "x must be (M, ", layer.K, ")");
    TORCH_CHECK(out.dim() == 2 && out.size(0) == x.size(0) && out.size(1) == layer.N, "out must be (M, ", layer.N, ")");
    const int M = (int)x.size(0), CH = 4096;
    const int chunk = M < CH ? M : CH;
    auto ws = torch::empty({(int64_t)cq_tlayer_gemm_workspace_bytes(&layer, chunk)}, blob.t.options());
    auto scratch = scratch_for(x.device());
    blob.use();
    uint8_t* sp = scratch.data_ptr<uint8_t>();
    const uint16_t* xp = (const uint16_t*)x.data_ptr();      // fp16 elements
    uint16_t* yp = (uint16_t*)out.data_ptr();
    for (int m0 = 0; m0 < M; m0 += CH) {
      const int rows = M - m0 < CH ? M - m0 : CH;
      const cq_tlayer* lp = &layer;
      void* y = yp + (size_t)m0 * layer.N;
      const int ldy = layer.N;
      check_status(cq_tlayers_gemm(&lp, 1, xp + (size_t)m0 * layer.K, layer.K, &y, &ldy, &bias, rows, accumulate ? 1 : 0, ws.data_ptr(),
                                   (uint32_t*)(sp + cq_scratch_bytes()), current_stream()),
                   "TileLayer.gemm");
    }
  }
};

// What a module's re-packed copies were made from: its four reference buffers, each by storage, address and version.
// The address alone does not identify a buffer (the allocator hands a freed block to the next tensor of that size, whose
// version is 0 again); the weak references keep the storages' records, so a recorded one is never taken for another.
struct BufferGuard {
  std::vector<c10::weak_intrusive_ptr<c10::StorageImpl>> storage;   // four entries
  std::array<const void*, 4> ptr{};
  std::array<uint64_t, 4> version{};

  // (tensors made under torch.inference_mode keep no version counter)
  static uint64_t version_of(const torch::Tensor& t) { return t.is_inference() ? 0u : (uint64_t)t._version(); }

  BufferGuard(torch::Tensor q, torch::Tensor s, torch::Tensor cw, torch::Tensor ci) {
    const torch::Tensor* t[4] = {&q, &s, &cw, &ci};
    for (int i = 0; i < 4; ++i) {
      storage.push_back(t[i]->storage().getWeakStorageImpl());
      ptr[i] = t[i]->const_data_ptr();
      version[i] = version_of(*t[i]);
    }
  }
  bool same(int i, const torch::Tensor& t) const {
    return t.has_storage() && t.storage().unsafeGetStorageImpl() == storage[i]._unsafe_get_target() &&
           t.const_data_ptr() == ptr[i] && version_of(t) == version[i];
  }
  bool holds(const torch::Tensor& q, const torch::Tensor& s, const torch::Tensor& cw, const torch::Tensor& ci) const {
    return same(0, q) && same(1, s) && same(2, cw) && same(3, ci);
  }
};

// QuantLinear.forward for a layer whose re-packed copies exist: checks that the module's reference buffers are still the
// ones the copies were made from, allocates the output and launches.  In Python these steps (four buffer look-ups, their
// addresses and versions, shapes, output, two calls) took 9 us of a 17 us call whose kernel runs for 4.
// A call of one row is bound by the host: with the output through the dispatcher, two views and the row layer's own checks
// (again) a 4096 x 4096 4-bit layer took 6.9 us a call, without them 5.7.
struct PackedForward {
  py::object row_ref, tile_ref, guard_ref;     // keep the copies and the record of their buffers alive
  RowLayer* row = nullptr;
  TileLayer* tile = nullptr;
  const BufferGuard* guard = nullptr;          // null: the buffers were released and nothing is compared
  int64_t K, N;
  int64_t row_rows, gemm_rows;                 // the row kernel takes 1 .. row_rows rows, the GEMM gemm_rows and more
  c10::Device device;
  uint32_t* status = nullptr;                  // the device's status word (scratch_for: kept for the process)

  static const std::array<PyObject*, 4>& names() {
    static const std::array<PyObject*, 4> n = {
        PyUnicode_InternFromString("qweight"), PyUnicode_InternFromString("scales"),
        PyUnicode_InternFromString("cherry_weight"), PyUnicode_InternFromString("cherry_indices")};
    return n;
  }
  static const torch::Tensor* buffer(const py::dict& buffers, int i) {
    PyObject* o = PyDict_GetItem(buffers.ptr(), names()[i]);
    return o && THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr;
  }

  // The ranges are the layer's, whichever copies exist: a call whose kernel has no copy yet is left to the general path.
  PackedForward(py::object row_layer, py::object tile_layer, py::object buffer_guard, int64_t row_rows_, int64_t gemm_rows_)
      : row_ref(std::move(row_layer)), tile_ref(std::move(tile_layer)), guard_ref(std::move(buffer_guard)),
        row_rows(row_rows_), gemm_rows(gemm_rows_), device(c10::kCPU) {
    if (!row_ref.is_none()) row = row_ref.cast<RowLayer*>();
    if (!tile_ref.is_none()) tile = tile_ref.cast<TileLayer*>();
    if (!guard_ref.is_none()) guard = guard_ref.cast<const BufferGuard*>();
    TORCH_CHECK(row || tile, "a layer without copies");
    K = row ? row->layer.K : tile->layer.K;
    N = row ? row->layer.N : tile->layer.N;
    device = (row ? row->blob : tile->blob).t.device();
    status = (uint32_t*)(scratch_for(device).data_ptr<uint8_t>() + cq_scratch_bytes());
  }

  // None: this call takes the general path
  c10::optional<torch::Tensor> forward(const torch::Tensor& x, const py::dict& buffers, const c10::optional<torch::Tensor>& bias) {
    if (!x.defined() || !x.is_cuda() || x.scalar_type() != torch::kFloat16 || x.dim() < 1 || x.size(-1) != K || x.numel() == 0 ||
        x.device() != device || !x.has_storage() || x.key_set().has(c10::DispatchKey::Python) || !x.is_contiguous() ||
        c10::impl::TorchDispatchModeTLS::any_modes_set())
      return c10::nullopt;
    const int64_t M = x.numel() / K;
    const bool by_row = M <= row_rows;
    if (by_row ? !row : (!tile || M < gemm_rows)) return c10::nullopt;
    for (int i = 0; i < 4 && guard; ++i) {
      const torch::Tensor* t = buffer(buffers, i);
      if (!t || !guard->same(i, *t)) return c10::nullopt;
    }
    c10::InferenceMode inference(true);        // as the decorated Python path
    const c10::cuda::CUDAGuard device_guard(device);
    c10::DimVector shape(x.sizes().begin(), x.sizes().end());
    shape.back() = N;
    // straight from the allocator (no dispatch mode is active: checked above), and the row kernel without views of rows
    torch::Tensor out = at::detail::empty_cuda(shape, torch::kFloat16, device, c10::nullopt);
    if (by_row) {
      row->blob.use();
      const cq_rlayer* lp = &row->layer;
      void* yp = out.mutable_data_ptr();
      check_status(cq_rlayers_matvec(&lp, 1, x.const_data_ptr(), (int)K, &yp, (int)N, (int)M, 0, status, current_stream()),
                   "RowLayer.matvec");
    } else {
      // 45 rows 5120 x 13824: 28.6 us with the bias in the GEMM, 32.4 with a kernel of its own
      const bool inside = bias.has_value() && bias->defined() && bias->scalar_type() == torch::kFloat16 && bias->device() == device &&
                          bias->dim() == 1 && bias->size(0) == N && bias->is_contiguous() && bias->has_storage() &&
                          !bias->key_set().has(c10::DispatchKey::Python);
      tile->gemm_bias(x.view({M, K}), out.view({M, N}), false, inside ? bias->const_data_ptr() : nullptr);
      if (inside) return out;
    }
    if (bias.has_value() && bias->defined()) out.add_(*bias);
    return out;
  }
};

// One launch (per four activation rows) for several row-tile layers that take the same activations
// (q / k / v, gate / up): outs[i] = [outs[i] +] x (M, K) fp16 . W_i^T.  The outputs are rows of `ldy`
// elements each: views into one (M, ldy) buffer, or separate (M, N_i) tensors when every N_i == ldy.
// norm_weight: the layers' input is the RMS norm of x (+ delta); the sum goes to `sum` (the last three may be undefined).
void row_layers_launch(const std::vector<RowLayer*>& layers, const torch::Tensor& x, const std::vector<torch::Tensor>& outs,
                       bool accumulate, const torch::Tensor& norm_weight, const torch::Tensor& delta, const torch::Tensor& sum,
                       double eps) {
  TORCH_CHECK(!layers.empty() && layers.size() <= 4 && layers.size() == outs.size(), "1 to 4 layers, one output each");
  const at::cuda::OptionalCUDAGuard device_guard(device_of(x));
  check_tensor(x, "x", torch::kFloat16, layers[0]->blob.t);
  const int K = layers[0]->layer.K;
  TORCH_CHECK(x.numel() % K == 0 && x.numel() > 0, "x must hold rows of ", K, " activations");
  const int M = (int)(x.numel() / K);
  const cq_rlayer* ls[4];
  void* ys[4];
  int64_t ldy = -1;
  for (size_t i = 0; i < layers.size(); ++i) {
    const auto& o = outs[i];
    TORCH_CHECK(o.is_cuda() && o.scalar_type() == torch::kFloat16 && o.device() == x.device() && o.dim() == 2 &&
                o.size(0) == M && o.size(1) == layers[i]->layer.N && o.stride(1) == 1,
                "out ", i, " must be a (", M, ", ", layers[i]->layer.N, ") fp16 CUDA tensor with unit column stride");
    if (M == 1) {
      ldy = std::max<int64_t>(ldy, o.size(1));          // a single row: the stride is never used
    } else {
      TORCH_CHECK(ldy < 0 || o.stride(0) == ldy, "the outputs must share one row stride (views of one buffer)");
      ldy = o.stride(0);
    }
    ls[i] = &layers[i]->layer;
    ys[i] = o.data_ptr();
  }
  for (const auto* l : layers) l->blob.use();
  auto scratch = scratch_for(x.device());
  uint32_t* status = (uint32_t*)(scratch.data_ptr<uint8_t>() + cq_scratch_bytes());
  if (norm_weight.defined()) {
    check_tensor(norm_weight, "norm_weight", torch::kFloat16, x);
    TORCH_CHECK(norm_weight.numel() == K, "norm_weight must hold ", K, " values");
    for (const auto* t : {&delta, &sum}) {
      if (!t->defined()) continue;
      check_tensor(*t, "delta / sum", torch::kFloat16, x);
      TORCH_CHECK(t->numel() == x.numel(), "delta and sum must have the shape of x");
    }
    check_status(cq_rlayers_matvec_norm(ls, (int)layers.size(), x.data_ptr(), delta.defined() ? delta.data_ptr() : nullptr,
                                        norm_weight.data_ptr(), (float)eps, sum.defined() ? sum.data_ptr() : nullptr, K, ys, (int)ldy, M,
                                        status, current_stream()),
                 "row_layers_matvec_norm");
    return;
  }
  check_status(cq_rlayers_matvec(ls, (int)layers.size(), x.data_ptr(), K, ys, (int)ldy, M, accumulate ? 1 : 0, status, current_stream()),
               "row_layers_matvec");
}
void row_layers_matvec(std::vector<RowLayer*> layers, torch::Tensor x, std::vector<torch::Tensor> outs, bool accumulate) {
  row_layers_launch(layers, x, outs, accumulate, torch::Tensor(), torch::Tensor(), torch::Tensor(), 0.0);
}
// The same on the RMS norm of x (+ delta), up to four rows; returns the sum x + delta (x itself without a delta).
torch::Tensor row_layers_matvec_norm(std::vector<RowLayer*> layers, torch::Tensor x, c10::optional<torch::Tensor> delta,
                                     torch::Tensor norm_weight, double eps, std::vector<torch::Tensor> outs) {
  torch::Tensor d, sum;
  if (delta.has_value()) {
    const at::cuda::OptionalCUDAGuard device_guard(device_of(x));
    d = *delta;
    sum = torch::empty_like(x);
  }
  row_layers_launch(layers, x, outs, false, norm_weight, d, sum, eps);
  return sum.defined() ? sum : x;
}

// TileLayer.gemm for layers that take the same activations (q / k / v, gate / up): one pre-pass and one launch per 4096
// rows.  Returns the outputs, (M, N_i) each.
std::vector<torch::Tensor> tile_layers_gemm(std::vector<TileLayer*> layers, torch::Tensor x) {
  TORCH_CHECK(!layers.empty() && layers.size() <= 4, "1 to 4 layers");
  const at::cuda::OptionalCUDAGuard device_guard(device_of(x));
  const cq_tlayer& first = layers[0]->layer;
  check_tensor(x, "x", torch::kFloat16, layers[0]->blob.t);
  TORCH_CHECK(x.dim() == 2 && x.size(1) == first.K && x.size(0) > 0, "x must be (M, ", first.K, ")");
  const int M = (int)x.size(0), n = (int)layers.size(), CH = 4096, chunk = M < CH ? M : CH;
  auto ws = torch::empty({(int64_t)cq_tlayers_gemm_workspace_bytes(&first, n, chunk)}, layers[0]->blob.t.options());
  auto scratch = scratch_for(x.device());
  std::vector<torch::Tensor> outs;
  const cq_tlayer* ls[4];
  void* ys[4];
  int ldys[4];
  for (int i = 0; i < n; ++i) {
    TORCH_CHECK(layers[i]->blob.t.device() == x.device(), "the layers must be on x's device");
    layers[i]->blob.use();
    ls[i] = &layers[i]->layer;
    ldys[i] = ls[i]->N;
    outs.push_back(torch::empty({M, ls[i]->N}, x.options()));
  }
  uint32_t* status = (uint32_t*)(scratch.data_ptr<uint8_t>() + cq_scratch_bytes());
  for (int m0 = 0; m0 < M; m0 += CH) {
    const int rows = M - m0 < CH ? M - m0 : CH;
    for (int i = 0; i < n; ++i) ys[i] = (uint16_t*)outs[i].data_ptr() + (size_t)m0 * ldys[i];
    check_status(cq_tlayers_gemm(ls, n, (const uint16_t*)x.data_ptr() + (size_t)m0 * first.K, first.K, ys, ldys, nullptr, rows, 0, ws.data_ptr(),
                                 status, current_stream()),
                 "tile_layers_gemm");
  }
  return outs;
}

// Reads and clears the status word the PreparedLayer launches report into.
bool device_timed_out(int device_index) {
  torch::Tensor t;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    auto it = g_scratch.find(device_index);
    if (it == g_scratch.end()) return false;
    t = it->second;
  }
  auto word = t.slice(0, (int64_t)cq_scratch_bytes(), (int64_t)cq_scratch_bytes() + 4).cpu();
  const bool bad = word.view(torch::kInt32).item<int32_t>() != 0;
  if (bad) t.zero_();
  return bad;
}

}  // namespace

// ---- element-wise kernels of the decode harness
std::vector<torch::Tensor> rmsnorm(torch::Tensor x, c10::optional<torch::Tensor> residual, torch::Tensor weight,
                                   double eps, bool return_sum) {
  const at::cuda::OptionalCUDAGuard device_guard(device_of(x));
  check_tensor(x, "x", torch::kFloat16, x);
  check_tensor(weight, "weight", torch::kFloat16, x);
  TORCH_CHECK(x.dim() == 2 && weight.numel() == x.size(1), "x must be (rows, hidden) and weight (hidden,)");
  const void* res = nullptr;
  if (residual.has_value()) {
    check_tensor(*residual, "residual", torch::kFloat16, x);
    TORCH_CHECK(residual->sizes() == x.sizes(), "residual must have the shape of x");
    res = residual->data_ptr();
  }
  auto y = torch::empty_like(x);
  torch::Tensor h;
  if (return_sum) h = torch::empty_like(x);
  check_status(cq_rmsnorm(x.data_ptr(), res, weight.data_ptr(), y.data_ptr(), return_sum ? h.data_ptr() : nullptr,
                          (int)x.size(0), (int)x.size(1), (float)eps, current_stream()),
               "rmsnorm");
  if (return_sum) return {y, h};
  return {y};
}

void rope_cache(torch::Tensor q, torch::Tensor k, torch::Tensor v, torch::Tensor cos_table, torch::Tensor sin_table,
                torch::Tensor positions, torch::Tensor k_cache, torch::Tensor v_cache) {
  const at::cuda::OptionalCUDAGuard device_guard(device_of(q));
  check_tensor(q, "q", torch::kFloat16, q);
  check_tensor(k, "k", torch::kFloat16, q);
  check_tensor(v, "v", torch::kFloat16, q);
  check_tensor(cos_table, "cos", torch::kFloat32, q);
  check_tensor(sin_table, "sin", torch::kFloat32, q);
  check_tensor(positions, "positions", torch::kInt64, q);
  check_tensor(k_cache, "k_cache", torch::kFloat16, q);
  check_tensor(v_cache, "v_cache", torch::kFloat16, q);
  TORCH_CHECK(q.dim() == 3 && k.dim() == 3 && v.sizes() == k.sizes() && q.size(0) == k.size(0) && q.size(2) == k.size(2),
              "q must be (T, H, D), k and v (T, KV, D)");
  const int T = (int)q.size(0), H = (int)q.size(1), KV = (int)k.size(1), D = (int)q.size(2);
  TORCH_CHECK(positions.numel() == T, "positions must have T entries");
  TORCH_CHECK(cos_table.dim() == 2 && cos_table.size(1) == D / 2 && sin_table.sizes() == cos_table.sizes(),
              "cos / sin tables must be (max_seq, D / 2)");
  // caches (max_seq, KV, D): the T tokens are one sequence; (B, max_seq, KV, D): T / B consecutive tokens per sequence
  TORCH_CHECK((k_cache.dim() == 3 || k_cache.dim() == 4) && v_cache.sizes() == k_cache.sizes(), "caches must be ([B,] max_seq, KV, D)");
  const int cd = (int)k_cache.dim();
  const int B = cd == 4 ? (int)k_cache.size(0) : 1;
  TORCH_CHECK(k_cache.size(cd - 2) == KV && k_cache.size(cd - 1) == D && k_cache.size(cd - 3) <= cos_table.size(0) && T % B == 0,
              "caches must be ([B,] max_seq, KV, D) with max_seq within the rotary tables and B dividing T");
  check_status(cq_rope_cache(q.data_ptr(), k.data_ptr(), v.data_ptr(), cos_table.data_ptr<float>(),
                             sin_table.data_ptr<float>(), (const long long*)positions.data_ptr(), k_cache.data_ptr(),
                             v_cache.data_ptr(), T, H, KV, D, (int)k_cache.size(cd - 3), T / B, current_stream()),
               "rope_cache");
}

torch::Tensor silu_mul(torch::Tensor gate, torch::Tensor up, bool full) {
  const at::cuda::OptionalCUDAGuard device_guard(device_of(gate));
  check_tensor(gate, "gate", torch::kFloat16, gate);
  check_tensor(up, "up", torch::kFloat16, gate);
  TORCH_CHECK(gate.sizes() == up.sizes(), "gate and up must have the same shape");
  auto out = torch::empty_like(gate);
  auto fn = full ? cq_silu_mul_full : cq_silu_mul;
  check_status(fn(gate.data_ptr(), up.data_ptr(), out.data_ptr(), (long long)gate.numel(), current_stream()), "silu_mul");
  return out;
}


torch::Tensor attn_decode(torch::Tensor q, torch::Tensor k_cache, torch::Tensor v_cache, torch::Tensor position) {
  const at::cuda::OptionalCUDAGuard device_guard(device_of(q));
  check_tensor(q, "q", torch::kFloat16, q);
  check_tensor(k_cache, "k_cache", torch::kFloat16, q);
  check_tensor(v_cache, "v_cache", torch::kFloat16, q);
  check_tensor(position, "position", torch::kInt64, q);
  // q (B, H, D), one query per sequence; caches (B, max_seq, KV, D), or (max_seq, KV, D) for B == 1
  TORCH_CHECK(q.dim() == 3, "q must be (B, H, D)");
  const int B = (int)q.size(0);
  const int cd = (int)k_cache.dim();
  TORCH_CHECK((cd == 4 && k_cache.size(0) == B) || (cd == 3 && B == 1), "caches must be (B, max_seq, KV, D)");
  TORCH_CHECK(k_cache.size(cd - 1) == q.size(2) && v_cache.sizes() == k_cache.sizes(), "caches must be ([B,] max_seq, KV, D)");
  TORCH_CHECK(position.numel() == B, "one position per sequence");
  auto out = torch::empty_like(q);
  // the ranges of a head meet in a per-device workspace (launches of one stream follow one another, which is how the
  // decode harness calls this)
  const size_t need = cq_attn_decode_workspace_bytes(B, (int)q.size(1), (int)q.size(2), (int)k_cache.size(cd - 3));
  torch::Tensor keep;
  void* ws = attn_workspace(q.device(), (size_t)B * q.size(1), need, &keep);
  check_status(cq_attn_decode(q.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), (const long long*)position.data_ptr(),
                              out.data_ptr(), B, (int)q.size(1), (int)k_cache.size(cd - 2), (int)q.size(2),
                              (int)k_cache.size(cd - 3), 1.0f / std::sqrt((float)q.size(2)), ws, current_stream()),
               "attn_decode");
  return out;
}

// A decode step: rope_cache of one token per sequence, then attn_decode (q and k may or may not be left rotated).
torch::Tensor attn_decode_step(torch::Tensor q, torch::Tensor k, torch::Tensor v, torch::Tensor cos_table, torch::Tensor sin_table,
                               torch::Tensor position, torch::Tensor k_cache, torch::Tensor v_cache) {
  const at::cuda::OptionalCUDAGuard device_guard(device_of(q));
  check_tensor(q, "q", torch::kFloat16, q);
  check_tensor(k, "k", torch::kFloat16, q);
  check_tensor(v, "v", torch::kFloat16, q);
  check_tensor(cos_table, "cos", torch::kFloat32, q);
  check_tensor(sin_table, "sin", torch::kFloat32, q);
  check_tensor(position, "position", torch::kInt64, q);
  check_tensor(k_cache, "k_cache", torch::kFloat16, q);
  check_tensor(v_cache, "v_cache", torch::kFloat16, q);
  TORCH_CHECK(q.dim() == 3 && k.dim() == 3 && v.sizes() == k.sizes() && q.size(0) == k.size(0) && q.size(2) == k.size(2),
              "q must be (B, H, D), k and v (B, KV, D)");
  const int B = (int)q.size(0), H = (int)q.size(1), KV = (int)k.size(1), D = (int)q.size(2);
  TORCH_CHECK(position.numel() == B, "one position per sequence");
  TORCH_CHECK(k_cache.dim() == 4 && k_cache.size(0) == B && k_cache.size(2) == KV && k_cache.size(3) == D && v_cache.sizes() == k_cache.sizes(),
              "caches must be (B, max_seq, KV, D)");
  const int S = (int)k_cache.size(1);
  TORCH_CHECK(cos_table.dim() == 2 && cos_table.size(1) == D / 2 && cos_table.size(0) >= S && sin_table.sizes() == cos_table.sizes(),
              "cos / sin tables must be (at least max_seq, D / 2)");
  auto out = torch::empty_like(q);
  torch::Tensor keep;
  void* ws = attn_workspace(q.device(), (size_t)B * H, cq_attn_decode_workspace_bytes(B, H, D, S), &keep);
  check_status(cq_attn_decode_step(q.data_ptr(), k.data_ptr(), v.data_ptr(), cos_table.data_ptr<float>(), sin_table.data_ptr<float>(),
                                   (const long long*)position.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), out.data_ptr(), B, H,
                                   KV, D, S, 1.0f / std::sqrt((float)D), ws, current_stream()),
               "attn_decode_step");
  return out;
}

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("vecquant3matmul_cherryq", &vecquant3matmul_cherryq, "a 3-bit version");
  m.def("vecquant4matmul_cherryq", &vecquant4matmul_cherryq, "a 4-bit version");
  m.def("Dequantize3Normal", &Dequantize3Normal, "Dequantize3Normal");
  m.def("Dequantize4Normal", &Dequantize4Normal, "Dequantize4Normal");
  m.def("pack", &pack, "GPU QuantLinear.pack");
  m.def("fake_quant", &fake_quant, "fake-quantised training weight");
  m.def("unpack_dense", &unpack_dense, "GPU QuantLinear.unpack");
  m.def("cache_clear", []() {
    check_status(cq_cache_clear(), "cache_clear");
    std::lock_guard<std::mutex> lock(g_guard_mu);
    g_guards.clear();
  });
  m.def("cache_stats", []() {
    int n = 0;
    uint64_t b = 0;
    cq_cache_stats(&n, &b);
    return std::make_pair(n, b);
  });
  m.def("rmsnorm", &rmsnorm, "RMSNorm with optional residual add");
  m.def("rope_cache", &rope_cache, "rotary embedding in place + KV cache write");
  m.def("silu_mul", &silu_mul, "silu(gate) * up", py::arg("gate"), py::arg("up"), py::arg("full") = false);
  m.def("attn_decode_step", &attn_decode_step, "rotary embedding, KV cache write and attention of a decode step");
  m.def("attn_decode", &attn_decode, "single-query attention over the KV cache");
  m.def("poll", []() { check_status(cq_poll(current_stream()), "poll"); });
  m.def("device_timed_out", &device_timed_out);
  m.def("row_layers_matvec", &row_layers_matvec, "one launch for row-tile layers sharing an activation row");
  m.def("tile_layers_gemm", &tile_layers_gemm, "one launch of the GEMM for tile layers sharing their activations");
  m.def("row_layers_matvec_norm", &row_layers_matvec_norm, "row_layers_matvec on the RMS norm of its input");
  m.def("abi_version", &cq_abi_version);
  py::class_<RowLayer>(m, "RowLayer")
      .def(py::init<torch::Tensor, torch::Tensor, torch::Tensor, torch::Tensor, int, int, int>())
      .def_static("supported", &RowLayer::supported)
      .def_static("row_limit", &RowLayer::row_limit)
      .def("matvec", &RowLayer::matvec)
      .def("matvec_gather", &RowLayer::matvec_gather)
      .def("matvec_swiglu", &RowLayer::matvec_swiglu)
      .def("unprepare", &RowLayer::unprepare)
      .def_property_readonly("blob", [](const RowLayer& p) { return p.blob.t; })
      .def_property_readonly("preferred_rows", [](const RowLayer& p) { return cq_rlayer_preferred_rows(&p.layer); })
      .def_property_readonly("out_features", [](const RowLayer& p) { return p.layer.N; })
      .def_property_readonly("in_features", [](const RowLayer& p) { return p.layer.K; });
  py::class_<TileLayer>(m, "TileLayer")
      .def(py::init<torch::Tensor, torch::Tensor, torch::Tensor, torch::Tensor, int, int, int>())
      .def("gemm", &TileLayer::gemm)
      .def_property_readonly("blob", [](const TileLayer& p) { return p.blob.t; });
  py::class_<BufferGuard>(m, "BufferGuard")
      .def(py::init<torch::Tensor, torch::Tensor, torch::Tensor, torch::Tensor>())
      .def("holds", &BufferGuard::holds);
  py::class_<PackedForward>(m, "PackedForward")
      .def(py::init<py::object, py::object, py::object, int64_t, int64_t>())
      .def("__call__", &PackedForward::forward);
  py::class_<PreparedLayer>(m, "PreparedLayer")
      .def(py::init<torch::Tensor, torch::Tensor, torch::Tensor, torch::Tensor, int, int, int>())
      .def(py::init<torch::Tensor, int, int, int, int, int>())
      .def("matvec", &PreparedLayer::matvec)
      .def("unprepare", &PreparedLayer::unprepare)
      .def_property_readonly("blob", [](const PreparedLayer& p) { return p.blob.t; })
      .def_property_readonly("bits", [](const PreparedLayer& p) { return p.layer.bits; })
      .def_property_readonly("in_features", [](const PreparedLayer& p) { return p.layer.K; })
      .def_property_readonly("out_features", [](const PreparedLayer& p) { return p.layer.N; })
      .def_property_readonly("num_cherries", [](const PreparedLayer& p) { return p.layer.C; })
      .def_property_readonly("group_size", [](const PreparedLayer& p) { return p.layer.G; });
}
