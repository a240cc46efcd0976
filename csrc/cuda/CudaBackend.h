// CUDA half of ProcessGroupCCL: owns the CudaComm (created lazily at the first CUDA collective,
// like the reference creates its communicators lazily, src/gpu/dpcpp_ccl.cpp:255-380), the
// communication stream, the stream fork/join and Work semantics (non-blocking wait = stream
// dependency, CCL_BLOCKING_WAIT = host poll with timeout, CCL_SAME_STREAM = run on the caller's
// stream; cf. src/gpu/dpcpp_ccl.cpp:382-472), the watchdog that turns device-side bounded-wait
// expiries into errors on the Work, and the NCCL point-to-point side channel.
#pragma once
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDAStream.h>

#include <functional>
#include <memory>
#include <mutex>

#include "cuda/CudaComm.h"
#include "pg/ProcessGroupCCL.hpp"

namespace ccl {

class NcclP2P;

// CUDA events are recycled through a process-wide pool: creating and destroying two or three
// events per collective costs more host time than launching the kernel.
struct PooledEvent {
  cudaEvent_t ev = nullptr;
  bool timing = false;
  int device = 0;
  ~PooledEvent();
  bool query() const { return cudaEventQuery(ev) == cudaSuccess; }
};
std::shared_ptr<PooledEvent> acquire_event(int device, bool timing);

class CudaBackendImpl {
 public:
  CudaBackendImpl(c10d::ProcessGroupCCL* pg, c10::intrusive_ptr<c10d::Store> store, int rank, int size);
  ~CudaBackendImpl();

  using LaunchFn = std::function<std::string(CudaComm&, cudaStream_t)>;  // returns the algorithm tag

  // Runs `fn` on the communication stream (or the current stream in same-stream mode) with the
  // proper event dependencies and returns the Work. `keep` tensors are kept alive until the caller
  // has waited for the work on the stream it was issued from, or the kernels have run.
  // `host_blocking`: wait() blocks the host until completion (barrier). `async_op` false: the caller
  // waits before it does anything else (`async_op=False` in torch.distributed), so the kernels go
  // straight onto its stream: no fork, no join, and the tensors need no keeping.
  c10::intrusive_ptr<c10d::Work> run(c10d::OpType type, const char* title, const at::Device& device,
                                     const LaunchFn& fn, const std::vector<at::Tensor>& keep,
                                     std::vector<at::Tensor> outs, std::vector<std::vector<at::Tensor>> nested,
                                     bool use_nested, uint64_t bytes, bool async_op = true, bool host_blocking = false);

  // NCCL p2p (send / recv, batched between start/endCoalescing).
  c10::intrusive_ptr<c10d::Work> p2p(bool is_send, at::Tensor& tensor, int peer, bool batched);
  void p2p_group_start();
  c10::intrusive_ptr<c10d::Work> p2p_group_end();
  bool p2p_batch_active() const { return p2p_batch_ops_ > 0; }

  CudaComm& comm(const at::Device& device);
  std::shared_ptr<CudaComm> comm_ptr(const at::Device& device);
  // Memory from the communicator's symmetric heap (see CudaComm::symm_alloc: collective in order).
  // The block goes back to the heap when the DataPtr / tensor dies; it keeps the communicator alive.
  c10::DataPtr symm_allocate(size_t bytes, const at::Device& device);
  at::Tensor symm_empty(int64_t numel, at::TensorOptions options);
  bool has_comm() const { return comm_ != nullptr; }
  c10::cuda::CUDAStream comm_stream(const at::Device& device);
  void shutdown();
  void abort();
  int status_code() const { return comm_ ? comm_->poll_status() : 0; }

 private:
  c10d::ProcessGroupCCL* pg_;
  c10::intrusive_ptr<c10d::Store> store_;
  int rank_, size_;
  std::mutex mu_;
  std::shared_ptr<CudaComm> comm_;
  std::unique_ptr<c10::cuda::CUDAStream> stream_;
  std::shared_ptr<PooledEvent> fork_event_;
  std::unique_ptr<NcclP2P> nccl_;
  int p2p_batch_ops_ = 0;
  bool p2p_in_group_ = false;
  std::vector<at::Tensor> p2p_batch_tensors_;
  at::Device p2p_device_{at::kCUDA, 0};
};

// The process-wide watchdog: keeps in-flight CUDA work alive until its end event fires, then
// finishes it (or fails it when the communicator reported a device-side timeout).
//
// It holds the Work weakly and the tensors through a KeepAlive that wait() may empty first: a program
// that enqueues faster than the GPU runs would otherwise find every temporary of every collective
// still owned by this thread, and the allocator growing until it has to synchronise and free.
class Watchdog {
 public:
  static Watchdog& get();
  struct KeepAlive {
    std::mutex mu;
    std::vector<at::Tensor> tensors;
    void drop() {
      std::vector<at::Tensor> gone;  // freed outside the lock
      std::lock_guard<std::mutex> g(mu);
      gone.swap(tensors);
    }
    // `stream` runs after the kernels: gives the tensors up in its order, whichever stream they were allocated for.
    void drop_after(c10::cuda::CUDAStream stream);
  };
  struct Item {
    c10::weak_intrusive_ptr<c10d::ProcessGroupCCL::AsyncWorkCCL> work;
    std::shared_ptr<PooledEvent> end;
    std::shared_ptr<CudaComm> comm;
    std::shared_ptr<KeepAlive> keep;       // null: nothing to keep
    cudaStream_t stream = nullptr;         // works of one stream complete in the order they were issued
    size_t flight_slot = 0;
    uint64_t seq = 0;
    std::chrono::milliseconds timeout{0};  // the group's timeout; 0 = no deadline (see Watchdog::retire)
    std::chrono::steady_clock::time_point since{};  // when this item came to the head of the queue
    bool raised = false;                   // the communicator has been told to abort
    Item() : work(c10::intrusive_ptr<c10d::ProcessGroupCCL::AsyncWorkCCL>()) {}
  };
  void enqueue(Item item);
  void drain();  // blocks until every queued work has completed
  void stop();

 private:
  Watchdog();
  void loop();
  static bool retire(std::deque<Item>& q);  // completes what has run; false if the head is still pending
  static void complete(Item& it, bool gave_up);
  std::mutex mu_;
  std::condition_variable cv_;
  std::deque<Item> q_;
  bool stop_ = false;
  bool busy_ = false;      // items taken out of q_ are not all retired yet
  bool asleep_ = false;    // the thread waits without a time limit: only then has enqueue() to wake it
  int drainers_ = 0;       // threads in drain()
  std::thread th_;
};

}  // namespace ccl
