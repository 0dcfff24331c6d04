// The common case of torch.ops.megabake.kv_attention / attention on the GPU without a line of Python.
//
// A call of either op through the Python registrations (ops.py, runtime.py) costs 25 to 40 us on the host, several times what
// a small launch takes.  Registered here for AutogradCUDA, ahead of them, is a path that checks its arguments, allocates the
// result and launches, 5 to 8 us.  Whatever is not plainly right (another dtype, shape, layout or device, a shape seen for
// the first time, a stream under capture, a status word that is set, an error from the launch) is passed on unchanged to those
// registrations, whose checks, errors and set-up it then gets.
#include <ATen/ATen.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

#include <mutex>
#include <vector>

#include "../../include/megabake_b200.h"

namespace {

using at::Tensor;

// The library's entry points, handed over with the handle: it is loaded by path, and this file links to nothing of it.
struct Entries {
  decltype(&mk_kv_attention_scratch) kv_attention;
  decltype(&mk_kv_attention_scratch_bytes) scratch_bytes;
  decltype(&mk_attention) attention;
};

// What the two launches of a decode attention share belongs to a stream (see runtime.py), for a few streams.
struct Scratch {
  cudaStream_t stream;
  int64_t batch;
  Tensor memory;
};
constexpr size_t kStreams = 8;

// What serves a head shape on a device.  Made once, never destroyed: its tensors would outlive the allocator.
struct Kernels {
  const int64_t heads, kv_heads, head_dim;
  const int device;
  std::mutex lock;  // of what follows, held for a call: calls of other shapes and devices go on beside it
  Entries entries{};
  mk_handle handle = nullptr;
  int64_t max_tokens = 0;
  const volatile int32_t* status = nullptr;  // pinned word a failed launch sets
  std::vector<Scratch> scratch;

  Kernels(int64_t heads, int64_t kv_heads, int64_t head_dim, int device) : heads(heads), kv_heads(kv_heads), head_dim(head_dim), device(device) {}
};

struct State {
  std::mutex lock;  // of the list, held for a look at it
  std::vector<Kernels*> known;  // one per shape and device, a handful
};
State& state() {
  static State* const s = new State;
  return *s;
}

Kernels* find(State& s, int64_t heads, int64_t kv_heads, int64_t head_dim, int device) {
  for (Kernels* k : s.known)
    if (k->heads == heads && k->kv_heads == kv_heads && k->head_dim == head_dim && k->device == device) return k;
  return nullptr;
}
Kernels* find(int64_t heads, int64_t kv_heads, int64_t head_dim, int device) {
  State& s = state();
  std::lock_guard<std::mutex> guard(s.lock);
  return find(s, heads, kv_heads, head_dim, device);
}

bool plain(const Tensor& t, at::ScalarType type, c10::Device device) {
  return t.defined() && t.scalar_type() == type && t.device() == device && t.layout() == at::kStrided;
}
bool is_shape(const Tensor& t, int64_t a, int64_t b, int64_t c, int64_t d) {
  return t.dim() == 4 && t.size(0) == a && t.size(1) == b && t.size(2) == c && t.size(3) == d;
}

// Each returns an undefined tensor where the call is not theirs.
Tensor kv_attention_now(const Tensor& source, const Tensor& key, const Tensor& value, const Tensor& key_cache, const Tensor& value_cache,
                        const Tensor& valid_length) {
  if (!source.defined() || !source.is_cuda() || source.dim() != 4 || source.size(1) != 1 || !key_cache.defined() || key_cache.dim() != 4) return {};
  const c10::Device device = source.device();
  const int64_t batch = source.size(0), heads = source.size(2), dim = source.size(3), capacity = key_cache.size(1), kv_heads = key_cache.size(2);
  if (batch < 1 || capacity < 1 || kv_heads < 1 || heads % kv_heads != 0 || capacity > INT32_MAX || batch > INT32_MAX) return {};
  for (const Tensor* t : {&source, &key, &value, &key_cache, &value_cache})
    if (!plain(*t, at::kBFloat16, device)) return {};
  if (!is_shape(key, batch, 1, kv_heads, dim) || !is_shape(value, batch, 1, kv_heads, dim) || !is_shape(key_cache, batch, capacity, kv_heads, dim) ||
      !is_shape(value_cache, batch, capacity, kv_heads, dim) || !key_cache.is_contiguous() || !value_cache.is_contiguous())
    return {};
  if (!plain(valid_length, at::kInt, device) || valid_length.dim() != 1 || valid_length.size(0) != 1 || !valid_length.is_contiguous()) return {};
  Kernels* const k = find(heads, kv_heads, dim, device.index());
  if (k == nullptr) return {};
  std::lock_guard<std::mutex> guard(k->lock);
  if (k->handle == nullptr || batch > k->max_tokens || *k->status != 0) return {};
  const c10::cuda::CUDAGuard on(device);
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return {};
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
  const Tensor q = source.contiguous(), kn = key.contiguous(), vn = value.contiguous();
  Tensor memory;
  for (size_t i = 0; i < k->scratch.size() && !memory.defined(); ++i)
    if (k->scratch[i].stream == stream) {
      if (k->scratch[i].batch >= batch) memory = k->scratch[i].memory;
      else k->scratch.erase(k->scratch.begin() + i);
    }
  if (!memory.defined()) {
    memory = at::empty({static_cast<int64_t>(k->entries.scratch_bytes(batch, heads, dim))}, source.options().dtype(at::kByte));
    if (k->scratch.size() >= kStreams) k->scratch.erase(k->scratch.begin());
    k->scratch.push_back({stream, batch, memory});
  }
  Tensor out = at::empty({batch * heads, 1, dim}, source.options());
  const int code = k->entries.kv_attention(k->handle, q.const_data_ptr(), kn.const_data_ptr(), vn.const_data_ptr(), key_cache.mutable_data_ptr(),
                                           value_cache.mutable_data_ptr(), static_cast<int32_t*>(valid_length.mutable_data_ptr()), static_cast<int>(batch),
                                           static_cast<int>(capacity), out.mutable_data_ptr(), memory.mutable_data_ptr(),
                                           static_cast<size_t>(memory.numel()), stream);
  return code == MK_OK ? out : Tensor();
}

Tensor attention_now(const Tensor& query, const Tensor& key, const Tensor& value, const std::optional<Tensor>& mask, double scale) {
  if (!query.defined() || !query.is_cuda() || query.dim() != 4 || !key.defined() || key.dim() != 4) return {};
  const c10::Device device = query.device();
  const int64_t batch = query.size(0), q_len = query.size(1), heads = query.size(2), dim = query.size(3), k_len = key.size(1), kv_heads = key.size(2);
  if (batch < 1 || q_len < 1 || k_len < 1 || kv_heads < 1 || heads % kv_heads != 0 || batch > INT32_MAX || q_len > INT32_MAX || k_len > INT32_MAX) return {};
  for (const Tensor* t : {&query, &key, &value})
    if (!plain(*t, at::kBFloat16, device)) return {};
  if (!is_shape(key, batch, k_len, kv_heads, dim) || !is_shape(value, batch, k_len, kv_heads, dim)) return {};
  const bool masked = mask.has_value() && mask->defined();
  if (masked && (!plain(*mask, at::kBFloat16, device) || !is_shape(*mask, batch, 1, q_len, k_len) || !mask->is_contiguous())) return {};
  Kernels* const k = find(heads, kv_heads, dim, device.index());
  if (k == nullptr) return {};
  std::lock_guard<std::mutex> guard(k->lock);
  if (k->handle == nullptr || *k->status == MK_STATUS_TIMEOUT) return {};
  const c10::cuda::CUDAGuard on(device);
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return {};
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
  const Tensor kk = key.contiguous(), vv = value.contiguous();
  Tensor q = query.contiguous();
  if (reinterpret_cast<uintptr_t>(q.const_data_ptr()) % 4) q = q.clone();  // begins at an odd element: the kernels read pairs
  Tensor out = at::empty({batch * heads, q_len, dim}, query.options());
  const int code = k->entries.attention(k->handle, q.const_data_ptr(), kk.const_data_ptr(), vv.const_data_ptr(), masked ? mask->const_data_ptr() : nullptr,
                                        static_cast<float>(scale), static_cast<int>(batch), static_cast<int>(q_len), static_cast<int>(k_len),
                                        out.mutable_data_ptr(), stream);
  return code == MK_OK ? out : Tensor();
}

// Whether what comes below autograd is the CUDA kernel at once: no fake or functional tensors, no modes, no other layer.
bool straight(c10::DispatchKeySet keys) {
  return (keys & c10::after_ADInplaceOrView_keyset).highestPriorityTypeId() == c10::DispatchKey::CUDA;
}

// Below autograd: the path above, or the Python registrations.
Tensor kv_attention_below(bool now, const Tensor& source, const Tensor& key, const Tensor& value, Tensor& key_cache, Tensor& value_cache, Tensor& valid_length) {
  if (now) {
    const at::AutoDispatchBelowADInplaceOrView below;
    const Tensor out = kv_attention_now(source, key, value, key_cache, value_cache, valid_length);
    if (out.defined()) {
      for (const Tensor* t : {&key_cache, &value_cache, &valid_length})
        if (!t->is_inference()) t->unsafeGetTensorImpl()->bump_version();
      return out;
    }
  }
  static const auto op = c10::Dispatcher::singleton()
                             .findSchemaOrThrow("megabake::kv_attention", "")
                             .typed<Tensor(const Tensor&, const Tensor&, const Tensor&, Tensor&, Tensor&, Tensor&)>();
  const at::AutoDispatchBelowAutograd below;
  return op.call(source, key, value, key_cache, value_cache, valid_length);
}
Tensor attention_below(bool now, const Tensor& query, const Tensor& key, const Tensor& value, const std::optional<Tensor>& mask, double scale) {
  if (now) {
    const at::AutoDispatchBelowADInplaceOrView below;
    const Tensor out = attention_now(query, key, value, mask, scale);
    if (out.defined()) return out;
  }
  static const auto op = c10::Dispatcher::singleton()
                             .findSchemaOrThrow("megabake::attention", "")
                             .typed<Tensor(const Tensor&, const Tensor&, const Tensor&, const std::optional<Tensor>&, double)>();
  const at::AutoDispatchBelowAutograd below;
  return op.call(query, key, value, mask, scale);
}

// Neither op has a derivative: results of inputs that want one say so when it is asked for.
struct KvAttention : torch::autograd::Function<KvAttention> {
  static Tensor forward(torch::autograd::AutogradContext*, bool now, const Tensor& source, const Tensor& key, const Tensor& value, Tensor key_cache,
                        Tensor value_cache, Tensor valid_length) {
    return kv_attention_below(now, source, key, value, key_cache, value_cache, valid_length);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext*, torch::autograd::variable_list) {
    TORCH_CHECK(false, "Trying to backward through megabake::kv_attention.default but no autograd formula was registered. "
                       "Please use register_autograd to add one.");
  }
};
struct Attention : torch::autograd::Function<Attention> {
  static Tensor forward(torch::autograd::AutogradContext*, bool now, const Tensor& query, const Tensor& key, const Tensor& value,
                        const std::optional<Tensor>& mask, double scale) {
    return attention_below(now, query, key, value, mask, scale);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext*, torch::autograd::variable_list) {
    TORCH_CHECK(false, "Trying to backward through megabake::attention.default but no autograd formula was registered. "
                       "Please use register_autograd to add one.");
  }
};

bool wants_grad(std::initializer_list<const Tensor*> tensors) {
  if (!c10::GradMode::is_enabled()) return false;
  for (const Tensor* t : tensors)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

Tensor kv_attention(c10::DispatchKeySet keys, const Tensor& source, const Tensor& key, const Tensor& value, Tensor& key_cache, Tensor& value_cache,
                    Tensor& valid_length) {
  if (wants_grad({&source, &key, &value, &key_cache, &value_cache, &valid_length}))
    return KvAttention::apply(straight(keys), source, key, value, key_cache, value_cache, valid_length);
  return kv_attention_below(straight(keys), source, key, value, key_cache, value_cache, valid_length);
}
Tensor attention(c10::DispatchKeySet keys, const Tensor& query, const Tensor& key, const Tensor& value, const std::optional<Tensor>& mask, double scale) {
  const Tensor none;
  if (wants_grad({&query, &key, &value, mask.has_value() ? &*mask : &none})) return Attention::apply(straight(keys), query, key, value, mask, scale);
  return attention_below(straight(keys), query, key, value, mask, scale);
}

}  // namespace

TORCH_LIBRARY_IMPL(megabake, AutogradCUDA, m) {
  m.impl("kv_attention", TORCH_FN(kv_attention));
  m.impl("attention", TORCH_FN(attention));
}

// From Python, when it has made (or replaced by a larger one) the handle for a head shape on a device.
extern "C" void megabake_ops_register(int64_t heads, int64_t kv_heads, int64_t head_dim, int device, int64_t max_tokens, void* handle,
                                      const int32_t* status, void* kv_attention_entry, void* scratch_bytes_entry, void* attention_entry) {
  State& s = state();
  Kernels* k;
  {
    std::lock_guard<std::mutex> guard(s.lock);
    k = find(s, heads, kv_heads, head_dim, device);
    if (k == nullptr) {
      k = new Kernels(heads, kv_heads, head_dim, device);
      k->status = status;
      s.known.push_back(k);
    }
  }
  std::lock_guard<std::mutex> guard(k->lock);
  k->entries.kv_attention = reinterpret_cast<decltype(&mk_kv_attention_scratch)>(kv_attention_entry);
  k->entries.scratch_bytes = reinterpret_cast<decltype(&mk_kv_attention_scratch_bytes)>(scratch_bytes_entry);
  k->entries.attention = reinterpret_cast<decltype(&mk_attention)>(attention_entry);
  k->handle = static_cast<mk_handle>(handle);
  k->max_tokens = max_tokens;
  k->status = status;
}
