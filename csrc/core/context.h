// Per-process description of one worker: who it is (WorkerInfo), where its cache tensors
// live, how to wait for a layer's KV to be produced, and which transports are usable.
// Role of kvtransfer/include/context.h:32-85 with one addition: device_id < 0 means the cache
// tensors are plain host memory (CPU plumbing without a GPU).
#pragma once
#include <atomic>
#include <memory>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "core/completion.h"
#include "core/types.h"

namespace kvx {

struct LayerInfo {
  size_t token_size;
  size_t block_size;
  uint64_t layer_addr;
  LayerInfo(size_t t, size_t b, uint64_t a) : token_size(t), block_size(b), layer_addr(a) {}
};

// Waits until the KV of `layer` has been produced on the device.
class ICudaBarrier {
 public:
  virtual void wait(uint32_t layer) = 0;
  // Raw cudaEvent_t of the layer (nullptr when the barrier is not event based); lets a device
  // transport order its stream after the layer without a host wait.
  virtual void* event(uint32_t layer) { (void)layer; return nullptr; }
  // Another process is about to be given the events.
  virtual void share() {}
  virtual ~ICudaBarrier() = default;
};

class NoCudaBarrier : public ICudaBarrier {
 public:
  void wait(uint32_t) override {}
};

// One event a layer.  With `peers` the caller's events serve until another process asks for them, and interprocess ones that are made
// then from there on: an interprocess event costs 1.2 us to record on the forward thread, a plain one 0.5, and a client that nobody
// pulls from is made sooner without (32 layers: 400 us instead of 500).
class CudaEventBarrier : public ICudaBarrier {
 public:
  explicit CudaEventBarrier(std::vector<uint64_t> events, bool peers = false, int device = -1)
      : events_(std::move(events)), peers_(peers), device_(device) {}
  ~CudaEventBarrier() override;
  void wait(uint32_t layer) override;
  // Asked for a layer that has been recorded: whoever knows that it was also sees which of its events that was.
  void* event(uint32_t layer) override {
    const std::vector<uint64_t>& ev = shared_.load(std::memory_order_acquire) ? peer_events_ : events_;
    return layer < ev.size() ? reinterpret_cast<void*>(ev[layer]) : nullptr;
  }
  // From here on the peer events are the layers' events; what the plain ones stand for so far is carried over.
  void share() override;
  // What the layer's latest record stands for has happened.
  bool ready(uint32_t layer);
  // Engine thread: layer event `event` (its plain one) on `stream`.
  void record(uint64_t event, uint64_t stream);

 private:
  bool make_peer_events();
  std::vector<uint64_t> events_, peer_events_;     // peer_events_: written before shared_ is set, not after
  const bool peers_;
  const int device_;
  std::unordered_map<uint64_t, uint64_t> peer_of_;
  std::mutex share_mu_;    // one share() at a time
  std::mutex mu_;          // record() against share()
  std::atomic<bool> shared_{false};
};

class Context {
 public:
  const InstanceId inst_name;
  const WorkerId worker_id;

  Context(const InstanceId& inst, WorkerId worker);
  Context(const Context&) = delete;

  void set_tp(uint32_t tp_size, uint32_t worker_tp_rank);
  void set_block_params(std::vector<size_t> block_sizes, std::vector<size_t> token_sizes,
                        uint32_t layer_num_blocks, uint32_t indexer_blk_ntpb = 0);
  void set_layer_info(int device_id, const std::vector<std::vector<LayerInfo>>& all_layer_infos);
  void set_cuda_barrier(std::unique_ptr<ICudaBarrier> barrier);
  void set_protocols(uint8_t mask) { worker_info_.transfer_protocols = mask; }

  WorkerInfo* worker_info_mutable() { return &worker_info_; }
  const WorkerInfo& worker_info() const { return worker_info_; }
  ICudaBarrier* cuda_barrier() { return barrier_.get(); }
  const std::vector<std::vector<LayerInfo>>& all_layer_infos() const { return layer_infos_; }
  const std::vector<std::vector<uint64_t>>& layer_data_address() const { return layer_addrs_; }
  // NVLink multicast addresses of the same tensors, when this worker's cache is a member of a multicast group
  // (a tensor-parallel decode group whose caches live in one symmetric allocation); empty otherwise.
  const std::vector<std::vector<uint64_t>>& multicast_address() const { return mc_addrs_; }
  void set_multicast_address(std::vector<std::vector<uint64_t>> a) { mc_addrs_ = std::move(a); }
  int device_id() const { return device_id_; }
  uint32_t num_layers() const { return worker_info_.num_layers; }
  uint32_t layer_num_blocks() const { return worker_info_.layer_num_blocks; }
  const std::vector<size_t>& block_sizes() const { return worker_info_.block_sizes; }
  bool supports(TransferProtocol::Kind k) const { return (worker_info_.transfer_protocols & k) != 0; }
  // Bytes of cache tensor `t` of any layer (block size x blocks): the bound every offset is checked against.
  size_t tensor_capacity(size_t t) const;
  InflightCounter& inflight() { return inflight_; }

 private:
  int device_id_{-1};
  WorkerInfo worker_info_;
  std::vector<std::vector<LayerInfo>> layer_infos_;
  std::vector<std::vector<uint64_t>> layer_addrs_;
  std::vector<std::vector<uint64_t>> mc_addrs_;
  std::unique_ptr<ICudaBarrier> barrier_;
  InflightCounter inflight_;
};

}  // namespace kvx
