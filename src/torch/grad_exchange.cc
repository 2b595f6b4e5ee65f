// Gradient hooks of DistributedOptimizer on one rank, in native code.
//
// A model hands over one gradient per parameter, hundreds per step, on the autograd thread.  A
// hook written in Python (a copy kernel into the gradient buffer, the priority queue, the launch)
// cost about 20 us each: 3.2 ms per step for the 161 tensors of ResNet-50, whose update takes the
// GPU 0.1 ms.  Here a hook takes the gradient tensor as it is (no kernel), and once enough is
// pending one call hands all of them to the update kernel, which reads every gradient where it
// lies, rounds it to the table's gradient type and updates the weights
// (psdev_dense_op_segs, include/ps/device/local_update.cuh).
//
// That read comes later than the hook and on another stream, so it is made only of memory that
// nobody else can write meanwhile (Private).  Autograd hands on a gradient without a copy as soon
// as its tensor has one owner, even where its storage has more: a custom backward may return views
// of a workspace that it writes again for the next layer.  Such a gradient is copied into the
// table's gradient buffer on the stream that made it, by the hook.
//
// The hooks sit on the parameters' gradient accumulators, next to hooks that a program registers
// on the parameters themselves, and run after those.  An accumulator belongs to the stream that was
// current when it was made and lives as long as the graphs that use it, so it is not held here: a
// tensor hook, which the parameter keeps, puts the hook on each new accumulator.  It stands behind
// the one for the program's tensor hooks, which Tensor::register_hook would drop.  (Held ones would
// keep accumulation on the stream of the constructor, out of reach of a graph capture.)
//
// A gradient stays alive until the kernel that reads it has finished: batches are kept with an
// event and dropped when it has fired, the rest when the step ends and the caller's stream has been
// ordered behind the kernels.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/function_hook.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <deque>
#include <mutex>
#include <optional>
#include <vector>

#include "ps/device/psdev.h"

namespace {

using torch::autograd::Node;
using torch::autograd::variable_list;
using SegsFn = int (*)(const psdev_world_t*, const psdev_table_t*, int, const psdev_seg_t*, int,
                       const psdev_opt_t*, int, int, void*);
using CopyFn = int (*)(const void*, int, void*, int, int64_t, void*);

class GradExchange {
 public:
  // `batch_elems`: gradients that a launch waits for, `busy_elems` while one is still running.
  // `world`, `table`, `opt`, `segs_fn`, `copy_fn`: addresses of the structures, of
  // psdev_dense_op_segs and of psdev_copy_cast;
  // `refresh` brings *opt up to date and is called before every launch.
  GradExchange(std::vector<at::Tensor> params, std::vector<int64_t> offsets,
               std::vector<int64_t> priorities, at::Tensor grad_buffer, uint64_t world,
               uint64_t table, uint64_t opt, uint64_t segs_fn, uint64_t copy_fn,
               uint64_t comm_stream, bool overlap, int64_t batch_elems, int64_t busy_elems,
               int64_t slice_elems, int channel, py::function refresh)
      : params_(std::move(params)),
        offsets_(std::move(offsets)),
        priorities_(std::move(priorities)),
        grad_buffer_(std::move(grad_buffer)),
        world_(reinterpret_cast<const psdev_world_t*>(world)),
        table_(reinterpret_cast<const psdev_table_t*>(table)),
        opt_(reinterpret_cast<const psdev_opt_t*>(opt)),
        segs_fn_(reinterpret_cast<SegsFn>(segs_fn)),
        copy_fn_(reinterpret_cast<CopyFn>(copy_fn)),
        device_(grad_buffer_.device().index()),
        overlap_(overlap),
        comm_(c10::cuda::getStreamFromExternal(reinterpret_cast<cudaStream_t>(comm_stream),
                                               device_)),
        batch_elems_(batch_elems),
        busy_elems_(busy_elems),
        slice_elems_(slice_elems),
        channel_(channel),
        refresh_(std::move(refresh)) {
    sent_.assign(params_.size(), kNotSent);
    hooks_.resize(params_.size());
    for (size_t i = 0; i < params_.size(); ++i) {
      TORCH_CHECK(params_[i].is_leaf() && params_[i].requires_grad(), "parameter ", i,
                  " is no leaf that takes a gradient");
      auto before = std::make_unique<BeforeAccumulation>(this, i);
      hooks_[i].tensor_hook = before.get();
      torch::autograd::impl::materialize_autograd_meta(params_[i])->hooks_.push_back(
          std::move(before));
    }
  }

  ~GradExchange() {
    py::gil_scoped_release no_gil;
    Detach();
  }

  void Detach() {
    for (size_t i = 0; i < hooks_.size(); ++i) {
      auto& of_tensor = torch::autograd::impl::materialize_autograd_meta(params_[i])->hooks_;
      of_tensor.erase(std::remove_if(of_tensor.begin(), of_tensor.end(),
                                     [&](const auto& h) {
                                       return h.get() == hooks_[i].tensor_hook;
                                     }),
                      of_tensor.end());
      if (auto node = hooks_[i].node.lock()) node->del_post_hook(hooks_[i].key);
    }
    hooks_.clear();
    std::lock_guard<std::mutex> lk(mu_);
    segs_.clear();
    pending_ = 0;
    held_.clear();
    OutliveComm();  // (without a step nobody waits for the launches)
    batches_.clear();
  }

  // End of a step: everything pending goes out, and the caller's stream waits for it.
  void Step() {
    std::unique_lock<std::mutex> lk(mu_);
    Drain(lk);
    const auto cur = at::cuda::getCurrentCUDAStream(device_);
    if (launched_on_) After(*launched_on_, cur);
    if (overlap_) {
      // Memory given back from here on is reused on the stream the gradients were made on; that
      // is `cur`, which now comes after the kernels, or the allocator is told.
      if (other_stream_ || (hook_stream_ && *hook_stream_ != cur)) OutliveComm();
    }
    while (!batches_.empty()) Retire();
    hook_stream_.reset();
    launched_on_.reset();
    other_stream_ = false;
    std::fill(sent_.begin(), sent_.end(), kNotSent);
  }

  int64_t launches() const { return launches_; }
  int64_t slices() const { return slices_; }
  int64_t staged() const { return staged_; }  // gradients that went through the gradient buffer

 private:
  struct Hook : torch::autograd::FunctionPostHook {
    Hook(GradExchange* owner, size_t index) : owner(owner), index(index) {}
    variable_list operator()(const variable_list& outputs, const variable_list& inputs) override {
      owner->Take(index, inputs);
      return outputs;
    }
    GradExchange* owner;
    size_t index;
  };
  struct BeforeAccumulation : torch::autograd::FunctionPreHook {
    BeforeAccumulation(GradExchange* owner, size_t index) : owner(owner), index(index) {}
    variable_list operator()(const variable_list& grads) override {
      owner->Attach(index);
      return grads;
    }
    GradExchange* owner;
    size_t index;
  };
  // Before a gradient is accumulated: the accumulator has the hook.
  void Attach(size_t i) {
    const auto node = torch::autograd::impl::try_get_grad_accumulator(params_[i]);
    if (!node || i >= hooks_.size() || hooks_[i].node.lock() == node) return;
    hooks_[i].key = node->add_post_hook(std::make_unique<Hook>(this, i));
    hooks_[i].node = node;
  }

  struct Batch {
    at::cuda::CUDAEvent read;  // the kernels that read the tensors have finished
    std::vector<at::Tensor> tensors;
  };

  static int DeviceType(at::ScalarType t) { return t == at::kFloat ? PSDEV_F32 : PSDEV_BF16; }

  // Whether `grad`, taken out of its parameter, is the only way to its memory.  The tensor that
  // autograd accumulated (`inputs`) is still alive here and may share the storage, and so may the
  // tensor that this one is a view of (the transpose of a matrix product, for a linear layer);
  // both go with the call that runs the hook.  Memory that is not the allocator's own may have
  // owners that torch does not know.
  static bool Private(const at::Tensor& grad, const variable_list& inputs) {
    const c10::Storage& mem = grad.storage();
    if (grad.use_count() != 1 ||
        mem.data_ptr().get_deleter() != c10::cuda::CUDACachingAllocator::get()->raw_deleter())
      return false;
    size_t owners = 1;
    for (const at::Tensor& x : inputs) {
      if (!x.defined() || !x.has_storage() || !x.storage().is_alias_of(mem)) continue;
      if (x.use_count() > 2) return false;  // (the engine's reference, and Python's if it has one)
      ++owners;
      if (x.is_view()) {
        if (x._base().use_count() > 1) return false;  // (the view's reference)
        ++owners;
      }
    }
    return mem.use_count() == owners;
  }

  // The gradient of parameter `i` into the table's gradient buffer, on the hook's stream: a kernel
  // of its own where the layout allows it (a fifth of what Tensor::copy_ costs this thread, less
  // than half of cudaMemcpyAsync).
  void Stage(size_t i, const at::Tensor& grad, bool plain, const c10::cuda::CUDAStream& cur) {
    ++staged_;
    const int64_t n = params_[i].numel();
    if (plain) {
      char* dst = static_cast<char*>(grad_buffer_.data_ptr()) +
                  offsets_[i] * grad_buffer_.element_size();
      const int rc = copy_fn_(grad.data_ptr(), DeviceType(grad.scalar_type()), dst,
                              DeviceType(grad_buffer_.scalar_type()), n, cur.stream());
      TORCH_CHECK(rc == 0, "psdev_copy_cast failed with ", rc);
    } else {
      at::NoGradGuard no_grad;
      grad_buffer_.narrow(0, offsets_[i], n).view(params_[i].sizes()).copy_(grad, true);
    }
  }

  // Parameter `i` has a gradient once more before the step ends (two backward passes): an update of
  // its own, after the one that the first gradient has made or will make.  Pieces of one launch
  // must not share a range, and the gradient buffer may still be read by the launch before.
  void Again(size_t i, const c10::cuda::CUDAStream& cur, std::unique_lock<std::mutex>& lk) {
    if (sent_[i] == kPending) Drain(lk);
    if (launched_on_) After(*launched_on_, cur);
  }

  // The memory of launched gradients is not used again before what runs on `comm_` has finished.
  void OutliveComm() {
    for (auto& b : batches_)
      for (auto& t : b.tensors)
        c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), comm_);
  }

  // Orders work on `next` behind what has been issued on `before`.
  void After(const c10::cuda::CUDAStream& before, const c10::cuda::CUDAStream& next) {
    if (before == next) return;
    fork_.record(before);
    fork_.block(next);
  }

  void Take(size_t i, const variable_list& inputs) {
    at::Tensor& slot = params_[i].mutable_grad();
    if (!slot.defined()) return;
    std::unique_lock<std::mutex> lk(mu_);
    const auto cur = at::cuda::getCurrentCUDAStream(device_);
    // (a launch comes behind the stream of its pieces: what another stream has made goes out first)
    if (!segs_.empty() && *pending_on_ != cur) Drain(lk);
    if (!hook_stream_) hook_stream_ = cur;
    else if (*hook_stream_ != cur) other_stream_ = true;
    const int64_t n = params_[i].numel(), padded = (n + 7) & ~int64_t(7);
    psdev_seg_t seg{};
    seg.begin = offsets_[i];
    seg.end = offsets_[i] + padded;
    seg.n_valid = offsets_[i] + n;
    seg.priority = priorities_[i];
    if (sent_[i] != kNotSent) Again(i, cur, lk);
    at::Tensor grad = std::move(slot);
    slot = at::Tensor();
    const auto dt = grad.scalar_type();
    const bool plain = grad.layout() == at::kStrided && grad.is_contiguous() && grad.is_cuda() &&
                       grad.device().index() == device_ && !grad.is_neg() &&
                       (dt == at::kFloat || dt == at::kBFloat16);
    if (plain && Private(grad, inputs)) {
      seg.src = grad.data_ptr();
      seg.dtype = DeviceType(dt);
      held_.push_back(std::move(grad));
    } else {
      Stage(i, grad, plain, cur);
    }
    segs_.push_back(seg);
    pending_on_ = cur;
    sent_[i] = kPending;
    pending_ += padded;
    slices_ += (padded + slice_elems_ - 1) / slice_elems_;
    if (pending_ >= batch_elems_) {
      const bool idle = Idle(cur);
      if (idle || pending_ >= busy_elems_) Drain(lk);
    }
  }

  // Gives up the gradients whose kernels have finished, and says whether all have.  While one is
  // running, what is pending would only queue up behind it; it goes out with what comes next
  // instead, in fewer and larger launches.  (An event's query takes this thread 1.4 us, so it is
  // made every 25 us at most: what is running at a look, or launched since, counts as running until
  // the next.  How often hardly matters: with 0, 10, 25, 50 and 100 us in between, a pass of
  // ResNet-50 took 1869, 1897, 1880, 1913 and 1845 us, of BERT-large 3412, 3406, 3385, 3408 and
  // 3349, each of them within 2 % of itself from run to run.)
  bool Idle(const c10::cuda::CUDAStream& cur) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    C10_CUDA_CHECK(cudaStreamIsCapturing(cur.stream(), &capture));
    if (capture != cudaStreamCaptureStatusNone) return true;  // (an event may not be queried)
    const auto now = std::chrono::steady_clock::now();
    if (!batches_.empty() && now < next_look_) return false;
    while (!batches_.empty() && batches_.front().read.query()) Retire();
    next_look_ = now + std::chrono::microseconds(25);
    return batches_.empty();
  }

  // Sends what is pending, behind the stream of its hooks.  `lk` holds mu_; it is given up while
  // Python runs, since a thread that has the interpreter lock may be waiting for mu_.
  void Drain(std::unique_lock<std::mutex>& lk) {
    if (segs_.empty()) return;
    lk.unlock();
    {
      py::gil_scoped_acquire gil;
      refresh_();
    }
    lk.lock();
    if (segs_.empty()) return;  // another thread has sent them
    const auto made_on = *pending_on_;
    const auto stream = overlap_ ? comm_ : made_on;
    After(made_on, stream);
    if (launched_on_) After(*launched_on_, stream);
    launched_on_ = stream;
    const int rc = segs_fn_(world_, table_, PSDEV_OP_PUSHPULL, segs_.data(),
                            static_cast<int>(segs_.size()), opt_, channel_, 0, stream.stream());
    TORCH_CHECK(rc == 0, "psdev_dense_op_segs failed with ", rc);
    launches_ += (segs_.size() + PSDEV_MAX_LOCAL_SEGS - 1) / PSDEV_MAX_LOCAL_SEGS;
    if (overlap_) {
      Batch b;
      if (!spare_.empty()) {
        b = std::move(spare_.back());
        spare_.pop_back();
      }
      b.tensors.swap(held_);
      b.read.record(comm_);
      batches_.push_back(std::move(b));
    }
    held_.clear();
    segs_.clear();
    pending_ = 0;
    for (auto& state : sent_)
      if (state == kPending) state = kLaunched;
  }

  void Retire() {
    Batch b = std::move(batches_.front());
    batches_.pop_front();
    b.tensors.clear();
    spare_.push_back(std::move(b));  // (its event is used again)
  }

  std::vector<at::Tensor> params_;
  std::vector<int64_t> offsets_, priorities_;
  at::Tensor grad_buffer_;
  const psdev_world_t* world_;
  const psdev_table_t* table_;
  const psdev_opt_t* opt_;
  SegsFn segs_fn_;
  CopyFn copy_fn_;
  c10::DeviceIndex device_;
  bool overlap_;
  c10::cuda::CUDAStream comm_;
  int64_t batch_elems_, busy_elems_, slice_elems_;
  int channel_;
  py::function refresh_;
  struct Attached {
    const torch::autograd::FunctionPreHook* tensor_hook = nullptr;
    std::weak_ptr<Node> node;  // the accumulator that has the hook, and the hook's key there
    uintptr_t key = 0;
  };
  std::vector<Attached> hooks_;

  enum Sent : char { kNotSent, kPending, kLaunched };
  std::vector<Sent> sent_;  // of each parameter in this step

  std::mutex mu_;
  std::vector<psdev_seg_t> segs_;
  std::vector<at::Tensor> held_;  // gradients of segs_
  std::deque<Batch> batches_;     // launched, not known to be finished
  std::vector<Batch> spare_;
  std::chrono::steady_clock::time_point next_look_{};  // not before
  at::cuda::CUDAEvent fork_;
  std::optional<c10::cuda::CUDAStream> pending_on_;   // hooks of what is pending ran here
  std::optional<c10::cuda::CUDAStream> launched_on_;  // launches of this step
  std::optional<c10::cuda::CUDAStream> hook_stream_;  // first hook of this step
  bool other_stream_ = false;                         // a later one ran elsewhere
  int64_t pending_ = 0;
  std::atomic<int64_t> launches_{0}, slices_{0}, staged_{0};
};

}  // namespace

void add_requests(py::module& m);  // requests.cc
void add_calls(py::module& m);     // calls.cc

PYBIND11_MODULE(psb200_torch, m) {
  add_requests(m);
  add_calls(m);
  using release = py::call_guard<py::gil_scoped_release>;
  py::class_<GradExchange>(m, "GradExchange")
      .def(py::init<std::vector<at::Tensor>, std::vector<int64_t>, std::vector<int64_t>, at::Tensor,
                    uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, bool, int64_t,
                    int64_t, int64_t, int, py::function>())
      .def("step", &GradExchange::Step, release())
      .def("detach", &GradExchange::Detach, release())
      .def_property_readonly("launches", &GradExchange::launches)
      .def_property_readonly("slices", &GradExchange::slices)
      .def_property_readonly("staged", &GradExchange::staged);
}
