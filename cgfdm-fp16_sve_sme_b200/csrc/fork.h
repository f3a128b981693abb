// Side streams for the launches of one RK stage: the surface, PML and interior
// launches write disjoint points and read none of each other's, so two of them
// branch off the caller's stream and join it again.  Under stream capture they
// become parallel branches of the graph.
#pragma once
#include <cuda_runtime.h>

#include <mutex>

namespace cgfdm {

// Whether `st` belongs to a partition of the SMs (a green context).  Work of
// side streams would run outside it.
bool stream_is_partitioned(cudaStream_t st);

struct ForkSet {
  int device = -1, priority = 0;
  cudaStream_t side[2] = {};
  cudaEvent_t start = nullptr, done[2] = {};
  cudaError_t create(int dev, int prio) {
    device = dev;
    priority = prio;
    cudaError_t e = cudaEventCreateWithFlags(&start, cudaEventDisableTiming);
    for (int q = 0; q < 2 && e == cudaSuccess; ++q) {
      e = cudaStreamCreateWithPriority(&side[q], cudaStreamNonBlocking, prio);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&done[q], cudaEventDisableTiming);
    }
    return e;
  }
  void destroy() {
    for (int q = 0; q < 2; ++q) {
      if (side[q]) cudaStreamDestroy(side[q]);
      if (done[q]) cudaEventDestroy(done[q]);
    }
    if (start) cudaEventDestroy(start);
    *this = ForkSet();
  }
};

// Idle sets whose owner went away, for the next owner (at most kForkIdle, the
// others are destroyed).  CUDA gives a stream its hardware queue at its first
// use, and a step's time depends on which queues the caller's stream and the
// two side streams got.  161x161x101 FP32, handles one after another: 0.68 to
// 0.72 ms a step (every other handle 0.77 in some processes) with side streams
// that stay, 0.76 in each with side streams of its own.  Creating and
// destroying a set takes 0.2 ms (4 ms the first time in a process).
constexpr int kForkIdle = 32;
class ForkPool {
 public:
  bool take(int device, int priority, ForkSet &out) {
    std::lock_guard<std::mutex> lk(mu_);
    for (int q = n_ - 1; q >= 0; --q)
      if (idle_[q].device == device && idle_[q].priority == priority) {
        out = idle_[q];
        idle_[q] = idle_[--n_];
        return true;
      }
    return false;
  }
  bool give(const ForkSet &s) {
    std::lock_guard<std::mutex> lk(mu_);
    if (n_ == kForkIdle) return false;
    idle_[n_++] = s;
    return true;
  }

 private:
  std::mutex mu_;
  ForkSet idle_[kForkIdle];
  int n_ = 0;
};
inline ForkPool g_fork_pool;

// The side streams of one owner (a handle or a batch, driven by one host
// thread at a time): a set for each priority that its callers' streams had.
class Fork {
 public:
  // The work that comes next branches off `st` of the current device.  The
  // side streams have the priority of `st`.  A stream of an SM partition gets
  // none, and its launches run in turn.
  cudaError_t attach(int device, cudaStream_t st) {
    at_ = -1;
    if (stream_is_partitioned(st)) return cudaSuccess;
    int prio = 0;
    cudaError_t e = cudaStreamGetPriority(st, &prio);
    if (e != cudaSuccess) return e;
    for (int q = 0; q < n_; ++q)
      if (sets_[q].priority == prio) {
        at_ = q;
        return cudaSuccess;
      }
    if (n_ == kPriorities) return cudaSuccess;
    if (!g_fork_pool.take(device, prio, sets_[n_])) {
      e = sets_[n_].create(device, prio);
      if (e != cudaSuccess) {
        sets_[n_].destroy();
        return e;
      }
    }
    at_ = n_++;
    return cudaSuccess;
  }
  // The owner's device is current.  A set with an error stays out of the pool.
  void destroy() {
    for (; n_ > 0; --n_) {
      ForkSet &s = sets_[n_ - 1];
      bool idle = true;
      for (int q = 0; q < 2; ++q) idle = cudaStreamSynchronize(s.side[q]) == cudaSuccess && idle;
      if (idle && g_fork_pool.give(s))
        s = ForkSet();
      else
        s.destroy();
    }
    at_ = -1;
  }
  const ForkSet *set() const { return at_ < 0 ? nullptr : &sets_[at_]; }

 private:
  static constexpr int kPriorities = 8;
  ForkSet sets_[kPriorities];
  int n_ = 0, at_ = -1;  // at_: the set of the stream that was attached last
};

// The branches of one stage off `st`, from begin() to join().  A function that
// leaves in between, on an error, still joins: `st` then waits for the work
// that the side streams have.  in_turn: everything runs on `st` itself.
class Branches {
 public:
  Branches(const Fork &f, cudaStream_t st, bool in_turn)
      : s_(in_turn ? nullptr : f.set()), st_(st) {}
  Branches(const Branches &) = delete;
  Branches &operator=(const Branches &) = delete;
  ~Branches() { join(); }
  cudaError_t begin() {
    if (!s_) return cudaSuccess;
    cudaError_t e = cudaEventRecord(s_->start, st_);
    for (int q = 0; q < 2 && e == cudaSuccess; ++q) {
      e = cudaStreamWaitEvent(s_->side[q], s_->start, 0);
      if (e == cudaSuccess) open_ = q + 1;
    }
    return e;
  }
  cudaError_t join() {
    cudaError_t first = cudaSuccess;
    for (int q = 0; q < open_; ++q) {
      cudaError_t e = cudaEventRecord(s_->done[q], s_->side[q]);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(st_, s_->done[q], 0);
      if (first == cudaSuccess) first = e;
    }
    open_ = 0;
    return first;
  }
  cudaStream_t side(int q) const { return s_ ? s_->side[q] : st_; }

 private:
  const ForkSet *s_;
  cudaStream_t st_;
  int open_ = 0;  // side streams that have branched off and not joined
};

}  // namespace cgfdm
