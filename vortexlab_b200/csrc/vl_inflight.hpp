// What the sims and batches of a process have in flight on each device.
//
// The resident step kernel takes the SMs that it needs for a whole call, and before other kernels: beside a
// batch, or three more sims, the two-kernel steps of all of them overlap instead. us per step of one sim, N sims
// stepping at once, resident / two-kernel (B200):
//   rig 442 x 84 FP64      N = 1 5.4 / 12.3, 2 5.4 / 6.8, 3 5.4 / 4.9, 4 5.4 / 3.8, 8 5.4 / 3.9
//   rig 882 x 166 FP64     N = 1 6.4 / 16.2, 2 6.4 / 8.5, 3 6.4 / 6.1, 4 6.4 / 5.5, 8 6.4 / 5.3
//   tank 482 x 242 FP32    N = 1 6.4 / 15.7, 2 6.4 / 8.6, 3 6.4 / 6.0, 4 6.4 / 4.9, 8 6.4 / 5.0
//   tank 742 x 372 FP64    N = 1 8.6 / 19.2, 2 8.6 / 11.0, 3 8.6 / 9.8, 4 8.6 / 9.0, 8 8.6 / 9.2
//   tank 1202 x 602 FP32   N = 1 11.6 / 23.0, 2 11.5 / 14.4, 3 11.5 / 12.5, 4 11.5 / 11.2, 8 11.5 / 11.4
//   2,000 steps of a batch of 24 tunnels (114 ms) beside a stepping tank of 482 x 242: 1,430 ms / 118 ms
// so for sims below kOverlapCells beside three more sims, and for all beside a batch.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>
#include <vector>

namespace vl {

constexpr size_t kOverlapCells = 200000;

// One sim's or batch's work; `end` is recorded behind the work of each call.
struct Work {
  int device = 0;
  cudaEvent_t end = nullptr;
  int weight = 1;         // of kMany
  int calls = 0;          // calls that are still queueing work
  bool queued = false;    // `end` has been recorded and not been seen to have passed
  static constexpr int kMany = 3;
};

class InFlight {
 public:
  static InFlight& of_process();
  void add(Work* w);
  void remove(Work* w);
  // A call of `w` that queues work. The end is recorded before finish().
  void start(Work* w);
  void finish(Work* w);
  // Whether the other sims and batches with work in flight on w's device weigh kMany or more (only those that do
  // so alone: `batches`).
  bool many_others(const Work* w, bool batches);

 private:
  std::mutex m_;
  std::vector<Work*> all_;
};

// A call that queues work, from its construction to the end of the scope.
class InFlightCall {
 public:
  explicit InFlightCall(Work* w) : w_(w) { InFlight::of_process().start(w_); }
  ~InFlightCall() { InFlight::of_process().finish(w_); }
  InFlightCall(const InFlightCall&) = delete;
  InFlightCall& operator=(const InFlightCall&) = delete;

 private:
  Work* w_;
};

}  // namespace vl
