#include "transport/device_stage.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <thread>

#include "core/envcfg.h"
#include "core/types.h"
#include "kernels/kvt_kernels.h"
#include "transport/copy_policy.h"

namespace kvx {

namespace {
std::atomic<uint64_t> g_memcpy_lists{0}, g_kernel_lists{0};
}

void copy_path_counters(uint64_t* memcpy_lists, uint64_t* kernel_lists) {
  *memcpy_lists = g_memcpy_lists.load();
  *kernel_lists = g_kernel_lists.load();
}

void cuda_check(int err, const char* what) {
  if (err != 0) {
    throw KVTransferException(ErrorKind::CUDA, std::string(what) + ": " +
                                                   cudaGetErrorString(static_cast<cudaError_t>(err)));
  }
}

PinnedBuffer::~PinnedBuffer() { release(); }

void PinnedBuffer::release() {
  if (host_ == nullptr) return;
  if (pinned_) cudaFreeHost(host_); else free(host_);
  host_ = nullptr;
  dev_ = 0;
  cap_ = 0;
}

char* PinnedBuffer::reserve(size_t bytes, bool pinned) {
  if (bytes <= cap_ && pinned == pinned_ && host_ != nullptr) return host_;
  release();
  size_t cap = std::max<size_t>(bytes, 4096);
  cap = (cap + (cap >> 2) + 4095) & ~size_t{4095};
  pinned_ = pinned;
  if (pinned) {
    void* h = nullptr;
    cuda_check(cudaHostAlloc(&h, cap, cudaHostAllocMapped | cudaHostAllocPortable), "cudaHostAlloc");
    void* d = nullptr;
    cuda_check(cudaHostGetDevicePointer(&d, h, 0), "cudaHostGetDevicePointer");
    host_ = static_cast<char*>(h);
    dev_ = reinterpret_cast<uint64_t>(d);
  } else {
    host_ = static_cast<char*>(malloc(cap));
    if (host_ == nullptr) throw std::bad_alloc();
  }
  cap_ = cap;
  return host_;
}

DeviceStage::DeviceStage(int device) : device_(device) {
  cuda_check(cudaSetDevice(device_), "cudaSetDevice");
  cudaStream_t s;
  cuda_check(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "cudaStreamCreate");
  stream_ = s;
  void* st = nullptr;
  cuda_check(cudaMalloc(&st, 16), "cudaMalloc(status)");
  d_status_ = static_cast<uint32_t*>(st);
  cuda_check(cudaMemsetAsync(d_status_, 0, 16, s), "cudaMemsetAsync");
  // the status words' copy, and the marks' records
  h_status_.reserve(kMarksAt + kMarks * sizeof(KvtCompletion), true);
  h_marks_ = reinterpret_cast<KvtCompletion*>(h_status_.data() + kMarksAt);
  d_marks_ = reinterpret_cast<KvtCompletion*>(h_status_.device_ptr() + kMarksAt);
  memset(h_marks_, 0, kMarks * sizeof(KvtCompletion));
}

DeviceStage::~DeviceStage() {
  cudaSetDevice(device_);
  if (stream_ != nullptr) {
    cudaStreamSynchronize(static_cast<cudaStream_t>(stream_));
    cudaStreamDestroy(static_cast<cudaStream_t>(stream_));
  }
  if (done_event_ != nullptr) cudaEventDestroy(static_cast<cudaEvent_t>(done_event_));
  if (d_triples_ != nullptr) cudaFree(d_triples_);
  if (d_status_ != nullptr) cudaFree(d_status_);
  if (staging_.data() != nullptr) cudaFree(staging_.data());
}

void* DeviceStage::record_done() {
  if (done_event_ == nullptr) {
    cudaEvent_t e;
    cuda_check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
    done_event_ = e;
  }
  cuda_check(cudaEventRecord(static_cast<cudaEvent_t>(done_event_), static_cast<cudaStream_t>(stream_)), "cudaEventRecord");
  return done_event_;
}

void DeviceStage::wait_event(void* event) {
  if (event == nullptr) return;
  cuda_check(cudaStreamWaitEvent(static_cast<cudaStream_t>(stream_), static_cast<cudaEvent_t>(event), 0),
             "cudaStreamWaitEvent");
}

// The list as copies of the copy engines, where the device's policy says so: one cudaMemcpyAsync per descriptor, bounds checked
// here.  False: the kernel is to take it.
bool DeviceStage::copy_engines(uint64_t src_base, uint64_t dst_base, const std::vector<Triple>& triples, uint64_t src_cap,
                               uint64_t dst_cap, int host_side) {
  if (host_side == HOST_NONE) return false;
  const size_t n = triples.size();
  size_t total = 0, min_len = SIZE_MAX;
  for (const Triple& t : triples) {
    total += t.len;
    min_len = std::min<size_t>(min_len, t.len);
  }
  const CopyDir dir = host_side == HOST_SRC ? CopyDir::H2D : CopyDir::D2H;
  if (CopyPolicy::get(device_).choose(dir, n, total, min_len) != CopyPath::MEMCPY) return false;
  for (size_t i = 0; i < n; i++) {
    const Triple& t = triples[i];
    if (t.src_off > src_cap || t.len > src_cap - t.src_off || t.dst_off > dst_cap || t.len > dst_cap - t.dst_off) {
      throw KVTransferException(ErrorKind::CUDA, "copy descriptor " + std::to_string(i) + " is out of bounds");
    }
    cuda_check(cudaMemcpyAsync(reinterpret_cast<void*>(dst_base + t.dst_off),
                               reinterpret_cast<const void*>(src_base + t.src_off), t.len, cudaMemcpyDefault,
                               static_cast<cudaStream_t>(stream_)),
               "cudaMemcpyAsync(block)");
  }
  memcpy_lists_++;
  g_memcpy_lists++;
  return true;
}

// Room for n descriptors; nothing that uses the present ones is running.
void DeviceStage::make_room(size_t n) {
  if (n <= d_cap_) return;
  if (d_triples_ != nullptr) cuda_check(cudaFree(d_triples_), "cudaFree");
  d_triples_ = nullptr;
  d_cap_ = 0;
  const size_t cap = std::max<size_t>(n + n / 2, 4096);
  void* p = nullptr;
  cuda_check(cudaMalloc(&p, cap * sizeof(Triple)), "cudaMalloc(triples)");
  d_triples_ = static_cast<uint64_t*>(p);
  h_triples_.reserve(cap * sizeof(Triple), true);
  d_cap_ = cap;
}

// Descriptors of all launches since the last sync stay resident: the pinned staging must not be overwritten while an upload is in
// flight, so grow-and-sync when it would not fit.
size_t DeviceStage::upload(const Triple* triples, size_t n) {
  if (used_ + n > d_cap_) {
    RTASSERT(kept_ == 0);      // forget() made room for the lists that are kept
    if (used_ > 0) sync();
    make_room(n);
  }
  static_assert(sizeof(Triple) == 24, "triples are 3 x u64");
  const size_t place = used_;
  char* h = h_triples_.data() + place * sizeof(Triple);
  memcpy(h, triples, n * sizeof(Triple));
  cuda_check(cudaMemcpyAsync(d_triples_ + place * 3, h, n * sizeof(Triple), cudaMemcpyHostToDevice, static_cast<cudaStream_t>(stream_)),
             "cudaMemcpyAsync(triples)");
  used_ += n;
  return place;
}

int DeviceStage::copy_grid(int grid_ctas, int host_side) const {
  if (grid_ctas > 0) return grid_ctas;
  // a copy with a host end is PCIe-bound: half a CTA per SM keeps the link full (measured 33 GB/s through the
  // SHM transport against 28 with two per SM) and leaves the SMs to the forward pass
  return std::max(1, static_cast<int>((host_side != HOST_NONE ? 0.5 : 2.0) * kvt_sm_count(device_) * env_kernel_copy_sm_usage()));
}

void DeviceStage::launch_list(uint64_t src_base, uint64_t dst_base, size_t place, size_t n, uint64_t src_cap, uint64_t dst_cap,
                              int grid_ctas, int host_side, bool cast) {
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  const size_t max_per_launch = env_kernel_copy_max_block_num();
  const int grid = copy_grid(grid_ctas, host_side);
  for (size_t off = 0; off < n; off += max_per_launch) {
    const uint32_t cnt = static_cast<uint32_t>(std::min(max_per_launch, n - off));
    const uint64_t* d = d_triples_ + (place + off) * 3;
    if (cast) {
      cuda_check(kvt_launch_copy_blocks_cast(src_base, dst_base, d, cnt, src_cap, dst_cap, d_status_, grid, s),
                 "kvt_launch_copy_blocks_cast");
    } else {
      cuda_check(kvt_launch_copy_blocks(src_base, dst_base, d, cnt, src_cap, dst_cap, d_status_, grid, s),
                 "kvt_launch_copy_blocks");
    }
  }
}

void DeviceStage::enqueue(uint64_t src_base, uint64_t dst_base, const std::vector<Triple>& triples, uint64_t src_cap,
                          uint64_t dst_cap, int grid_ctas, int host_side, bool cast_bf16_e4m3) {
  if (triples.empty()) return;
  cuda_check(cudaSetDevice(device_), "cudaSetDevice");
  if (!cast_bf16_e4m3 && copy_engines(src_base, dst_base, triples, src_cap, dst_cap, host_side)) return;
  kernel_lists_++;
  g_kernel_lists++;
  launch_new(src_base, dst_base, triples.data(), triples.size(), src_cap, dst_cap, grid_ctas, host_side, cast_bf16_e4m3);
}

// A list that is used once: a short one travels in the launch's parameters, any other is uploaded first.  The upload is a copy of the
// engine that also brings the blobs, so it would wait behind the one under way, and its own blob behind it.
void DeviceStage::launch_new(uint64_t src_base, uint64_t dst_base, const Triple* triples, size_t n, uint64_t src_cap, uint64_t dst_cap,
                             int grid_ctas, int host_side, bool cast) {
  if (!cast && n <= std::min<size_t>(KVT_CARRIED_DESCS, env_kernel_copy_max_block_num())) {
    cuda_check(kvt_launch_copy_blocks_carried(src_base, dst_base, reinterpret_cast<const uint64_t*>(triples), static_cast<uint32_t>(n),
                                              src_cap, dst_cap, d_status_, copy_grid(grid_ctas, host_side), stream_),
               "kvt_launch_copy_blocks_carried");
    return;
  }
  const size_t place = upload(triples, n);
  launch_list(src_base, dst_base, place, n, src_cap, dst_cap, grid_ctas, host_side, cast);
}

// The bytes of a list whose source is one dense run that is worth staging; 0 for any other.
uint64_t DeviceStage::dense_source(const std::vector<Triple>& triples, uint64_t src_cap) {
  uint64_t total = 0;
  for (const Triple& t : triples) {
    if (t.src_off != triples[0].src_off + total) return 0;
    total += t.len;
  }
  const uint64_t first = triples[0].src_off;
  return total < kStagingLeast || total > env_staging_bytes() || first > src_cap || total > src_cap - first ? 0 : total;
}

bool DeviceStage::reserve_staging(size_t bytes) {
  if (bytes > env_staging_bytes()) return false;     // a blob is staged whole or not at all
  cuda_check(cudaSetDevice(device_), "cudaSetDevice");
  return staging_.reserve(
      bytes,
      [](size_t n) {
        void* p = nullptr;
        if (cudaMalloc(&p, n) == cudaSuccess) return p;
        cudaGetLastError();      // no room: the lists go through the mapping
        return static_cast<void*>(nullptr);
      },
      [this](void* smaller) {
        cudaStreamSynchronize(static_cast<cudaStream_t>(stream_));
        cudaFree(smaller);
      });
}

// A copy engine brings host memory at 55.3 GB/s where the loads of the SMs reach 51.1, and beside SM stores in the other direction, as
// on a GPU that is sender and receiver, 38 GB/s each way against 35 (4 MiB a copy).  It wants long runs (1 MiB 44.5 GB/s, 64 KiB 12):
// a frame's blob is one and a layer's pages are not, hence one copy of the blob into a buffer on this GPU and a kernel from there to
// the pages (4 MiB: 5 us).  The buffer holds the whole blob or is not used: in pieces of 8 MiB, each copied when the one before had been
// scattered, 32 MiB a layer took 37.0 ms a step, through the mapping 30.1, whole 27.1 (16 MiB: 17.8, 14.9, 14.9).
void DeviceStage::enqueue_from_host(uint64_t src_base, uint64_t dst_base, const std::vector<Triple>& triples, uint64_t src_cap,
                                    uint64_t dst_cap) {
  if (triples.empty()) return;
  cuda_check(cudaSetDevice(device_), "cudaSetDevice");
  if (copy_engines(src_base, dst_base, triples, src_cap, dst_cap, HOST_SRC)) return;
  kernel_lists_++;
  g_kernel_lists++;
  const uint64_t total = dense_source(triples, src_cap);
  if (total == 0 || !reserve_staging(total)) {
    launch_new(src_base, dst_base, triples.data(), triples.size(), src_cap, dst_cap, 0, HOST_SRC, false);
    return;
  }
  const uint64_t from = triples[0].src_off;
  cuda_check(cudaMemcpyAsync(staging_.data(), reinterpret_cast<const void*>(src_base + from), total, cudaMemcpyDefault,
                             static_cast<cudaStream_t>(stream_)),
             "cudaMemcpyAsync(staging)");
  std::vector<Triple> local(triples);
  for (Triple& t : local) t.src_off -= from;
  launch_new(reinterpret_cast<uint64_t>(staging_.data()), dst_base, local.data(), local.size(), total, dst_cap, 0, HOST_NONE, false);
}

void DeviceStage::forget(size_t lists_total) {
  RTASSERT(waited_ == marks_);
  cuda_check(cudaSetDevice(device_), "cudaSetDevice");
  used_ = kept_ = 0;
  make_room(lists_total);
}

size_t DeviceStage::keep(const std::vector<Triple>& triples) {
  if (triples.empty()) return 0;
  cuda_check(cudaSetDevice(device_), "cudaSetDevice");
  const size_t place = upload(triples.data(), triples.size());
  kept_ = used_;
  return place;
}

void DeviceStage::enqueue_kept(uint64_t src_base, uint64_t dst_base, size_t place, const std::vector<Triple>& triples, uint64_t src_cap,
                               uint64_t dst_cap, int host_side, bool cast_bf16_e4m3) {
  if (triples.empty()) return;
  cuda_check(cudaSetDevice(device_), "cudaSetDevice");
  if (!cast_bf16_e4m3 && copy_engines(src_base, dst_base, triples, src_cap, dst_cap, host_side)) return;
  kernel_lists_++;
  g_kernel_lists++;
  launch_list(src_base, dst_base, place, triples.size(), src_cap, dst_cap, 0, host_side, cast_bf16_e4m3);
}

uint64_t DeviceStage::mark() {
  RTASSERT(marks_ - waited_ < kMarks);
  cuda_check(kvt_launch_complete(d_status_, d_marks_ + (marks_ + 1) % kMarks, marks_ + 1, stream_), "kvt_launch_complete");
  return ++marks_;
}

bool DeviceStage::poll_mark(uint64_t m) {
  RTASSERT(m == waited_ + 1 && m <= marks_);
  KvtCompletion* rec = h_marks_ + m % kMarks;
  if (__atomic_load_n(&rec->seq, __ATOMIC_ACQUIRE) != m) {
    if (++polls_ % 1024 != 0) return false;
    // a stream that failed never writes the record, and one that has run dry has written it
    const cudaError_t e = cudaStreamQuery(static_cast<cudaStream_t>(stream_));
    if (e == cudaErrorNotReady) {
      cudaGetLastError();
      return false;
    }
    if (__atomic_load_n(&rec->seq, __ATOMIC_ACQUIRE) != m) {
      cuda_check(e, "cudaStreamQuery");
      throw KVTransferException(ErrorKind::CUDA, "a copy ended without its record");
    }
  }
  waited_ = m;
  if (waited_ == marks_) used_ = kept_;
  if (rec->status != 0) {
    throw KVTransferException(ErrorKind::CUDA, "copy kernel rejected descriptor " + std::to_string(rec->detail) + " (status " +
                                                   std::to_string(rec->status) + ")");
  }
  return true;
}

void DeviceStage::wait_mark(uint64_t m) {
  for (uint32_t spins = 0; !poll_mark(m); ++spins) {
    if (spins < 4096) std::this_thread::yield(); else std::this_thread::sleep_for(std::chrono::microseconds(5));
  }
}

void DeviceStage::quiesce() noexcept { cudaStreamSynchronize(static_cast<cudaStream_t>(stream_)); }

void DeviceStage::launch_resident(uint64_t src_base, uint64_t dst_base, const uint64_t* d_triples, size_t n,
                                  uint64_t src_cap, uint64_t dst_cap, int grid_ctas, uint32_t* status) {
  if (n == 0) return;
  uint32_t* st = status != nullptr ? status : d_status_;
  cuda_check(cudaSetDevice(device_), "cudaSetDevice");
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  const size_t max_per_launch = env_kernel_copy_max_block_num();
  int grid = grid_ctas;
  if (grid <= 0) grid = std::max(1, static_cast<int>(2 * kvt_sm_count(device_) * env_kernel_copy_sm_usage()));
  for (size_t off = 0; off < n; off += max_per_launch) {
    const uint32_t cnt = static_cast<uint32_t>(std::min(max_per_launch, n - off));
    cuda_check(kvt_launch_copy_blocks(src_base, dst_base, d_triples + off * 3, cnt, src_cap, dst_cap, st, grid, s),
               "kvt_launch_copy_blocks");
  }
}

void DeviceStage::sync() {
  cuda_check(cudaSetDevice(device_), "cudaSetDevice");
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  cuda_check(cudaMemcpyAsync(h_status_.data(), d_status_, 8, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync(status)");
  cuda_check(cudaStreamSynchronize(s), "cudaStreamSynchronize");
  used_ = kept_;
  uint32_t st[2];
  memcpy(st, h_status_.data(), 8);
  if (st[0] != 0) {
    cudaMemsetAsync(d_status_, 0, 16, s);
    throw KVTransferException(ErrorKind::CUDA, "copy kernel rejected descriptor " + std::to_string(st[1]) +
                                                   " (status " + std::to_string(st[0]) + ")");
  }
}

}  // namespace kvx
