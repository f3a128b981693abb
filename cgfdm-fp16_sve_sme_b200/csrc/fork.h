// Side streams for the launches of one RK stage: the surface, PML and interior
// launches write disjoint points and read none of each other's, so two of them
// branch off the caller's stream and join it again.  Under stream capture they
// become parallel branches of the graph.
#pragma once
#include <cuda_runtime.h>

namespace cgfdm {

// Whether `st` belongs to a partition of the SMs (a green context).  Work of
// side streams would run outside it.
bool stream_is_partitioned(cudaStream_t st);

struct ForkSet {
  int priority = 0;
  cudaStream_t side[2] = {};
  cudaEvent_t start = nullptr, done[2] = {};
  cudaError_t create(int prio) {
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

// The side streams of one owner (a handle or a batch, driven by one host
// thread at a time): a set for each priority that its callers' streams had,
// which takes 0.1 ms to create and as long to destroy (4 ms the first time in
// a process).
class Fork {
 public:
  // The work that comes next branches off `st` (of the current device).  The
  // side streams have the priority of `st`.  A stream of an SM partition gets
  // none, and its launches run in turn.
  cudaError_t attach(cudaStream_t st) {
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
    e = sets_[n_].create(prio);
    if (e != cudaSuccess) {
      sets_[n_].destroy();
      return e;
    }
    at_ = n_++;
    return cudaSuccess;
  }
  void destroy() {
    while (n_ > 0) sets_[--n_].destroy();
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
