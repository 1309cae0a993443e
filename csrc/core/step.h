// Layer-ready pipeline of one engine step.
//
// A Step carries two monotone counters that sender threads block on:
//   recorded(i): the engine has *recorded* the CUDA event of layer i on its forward stream
//                (host-side fact).  A device transport may now order its own stream after
//                that event and enqueue the layer's transfer without any host wait.
//   ready(i):    the event of layer i has *completed* (the KV bytes exist).  Host-driven
//                transports (TCP, shared memory) wait for this before they read the cache.
// StepGuard is the engine-side handle: the forward thread calls after_record_one() per layer,
// a wait-layers thread turns completed events into ready(i).  Same protocol as the
// reference's Step/StepGuard (kvtransfer/src/step.cpp:42-81), plus the recorded counter.
#pragma once
#include <atomic>
#include <memory>
#include <vector>

#include "core/context.h"
#include "core/util.h"

namespace kvx {

class Step {
 public:
  const size_t step_idx;
  const Timepoint start_send_ts = SteadyClock::now();
  std::vector<int64_t> sub_queue_time_us;  // written by whoever submits: the engine thread, or the target manager's under its lock
  Timepoint flush_send_ts;                 // written by the engine thread
  Timepoint wait_layers_start_ts;          // written by the wait-layers thread
  Timepoint wait_layers_end_ts;
  bool frozen = false;                     // born with every layer complete (freeze / migration steps)

  explicit Step(size_t idx) : step_idx(idx) {}
  ~Step();

  void wait_layer_ready(uint32_t layer) { want_ready(); data_signal_.wait(layer); }
  bool layer_ready(uint32_t layer) { return data_signal_.value() > layer; }
  bool wait_layer_ready_for(uint32_t layer, std::chrono::milliseconds d) { want_ready(); return data_signal_.wait_for(layer, d); }
  // A host-driven transport is going to follow ready(i) layer by layer.  Without it the wait-layers thread sleeps until
  // every layer has been recorded and then waits for the last event alone: its waits for the others would contend for
  // the driver with the forward thread's event records and the sender's launches, for nobody.
  void want_ready() {
    if (!ready_wanted_.exchange(true, std::memory_order_acq_rel)) record_signal_.kick();
  }
  // wait-layers thread: true when all `layers` have been recorded before anybody wanted ready(i), and the last of their
  // events implies the others
  bool all_recorded_unwanted(uint32_t layers) {
    return !ready_wanted_.load(std::memory_order_acquire) && record_signal_.wait_or(layers - 1, ready_wanted_) &&
           !ready_wanted_.load(std::memory_order_acquire) && last_event_implies(layers);
  }
  uint32_t notify_layer_ready(uint32_t layers_done) { return data_signal_.release(layers_done); }
  void wait_layer_recorded(uint32_t layer) { record_signal_.wait(layer); }
  uint32_t notify_layer_recorded(uint32_t layers_recorded) { return record_signal_.release(layers_recorded); }
  void notify_one_recorded() { record_signal_.release(); }
  // The raw handle of the stream that the next layer's event was recorded on, said before notify_one_recorded().  Only the
  // engine thread calls it.
  void note_stream(uint64_t stream) {
    const uint32_t n = in_line_.load(std::memory_order_relaxed);
    if (n == 0) stream_ = stream;
    if (stream != stream_) out_of_line_ = true;
    if (!out_of_line_) in_line_.store(n + 1, std::memory_order_release);
  }
  void note_unknown_stream() { out_of_line_ = true; }
  // A frozen step records nothing itself: the events it is ordered behind are those of the steps before it.
  void take_in_line(uint32_t layers) { in_line_.store(layers, std::memory_order_release); }
  // True: the events of layers [0, layers) were all recorded in this step (for a frozen step: in the last one that recorded
  // any) and follow one another on one stream, so that the last one implies the others.  False where that is not known: after a flush that came before the last layer's record, the
  // event of a layer that was not recorded is one of an earlier step and says nothing about this one.
  bool last_event_implies(size_t layers) const { return in_line_.load(std::memory_order_acquire) >= layers; }
  uint32_t layers_recorded() { return record_signal_.value(); }

  Timepoint last_send_finish_ts() const noexcept { return Timepoint(SteadyClock::duration(last_send_finish_.load())); }
  void update_last_send_finish_ts(Timepoint t) noexcept;

 private:
  SyncSemaphore data_signal_;
  SyncSemaphore record_signal_;
  std::atomic<bool> ready_wanted_{false};
  uint64_t stream_{0};
  bool out_of_line_{false};             // engine thread: a layer came on another stream, or on one that was not named
  std::atomic<uint32_t> in_line_{0};    // leading layers noted on one stream
  std::atomic<int64_t> last_send_finish_{0};
};

class StepGuard {
 public:
  const uint32_t num_layers;
  StepGuard(uint32_t layers, ICudaBarrier* barrier, std::shared_ptr<Step> step);
  StepGuard(Context* ctx, std::shared_ptr<Step> step);

  size_t step_id() const { return step_->step_idx; }
  std::shared_ptr<Step>& step() { return step_; }
  void wait_layers();        // runs on the wait-layers thread
  void after_record_one();   // engine thread: one more layer event recorded
  void after_record_all();
  void layer_ready_all();    // flush: everything recorded (events still gate readiness)

 private:
  std::shared_ptr<Step> step_;
  ICudaBarrier* barrier_;
};

}  // namespace kvx
