// Book-keeping of the attention calls' status words, plain C++ (no CUDA, no torch).
//
// A call claims a slot, whose word reads kPending until the GPU has stored the call's status there, and then
// says whether it launched what stores it.  Calls of several threads and streams are under way at the
// same time: their words arrive in any order, and a slot that is claimed but not launched yet neither counts as
// arrived nor is handed out again.
#pragma once
#include <cstdint>
#include <mutex>

namespace fmb {

class StatusRing {
 public:
  static constexpr int kSlots = 256, kPending = -1;
  struct Failure {
    int code;            // 0: none
    const char* what;
  };

  explicit StatusRing(volatile int* words) : words_(words) {}
  volatile int* word(int slot) { return words_ + slot; }

  // a free slot, its word pending; -1: every slot is in use
  int claim(const char* what, int device) {
    std::lock_guard<std::mutex> lock(mu_);
    for (int n = 0; n < kSlots; ++n) {
      const uint64_t at = head_ + n;
      Slot& s = slots_[at % kSlots];
      if (s.state != kFree) continue;
      head_ = at + 1;
      words_[at % kSlots] = kPending;
      s = Slot{kClaimed, device, what, at};
      return (int)(at % kSlots);
    }
    return -1;
  }
  // the word of the slot's call will come
  void launched(int slot) {
    std::lock_guard<std::mutex> lock(mu_);
    slots_[slot].state = kLaunched;
  }
  // the slot's call launched nothing
  void withdraw(int slot) {
    std::lock_guard<std::mutex> lock(mu_);
    slots_[slot].state = kFree;
  }
  // frees the slots whose words have arrived, in the order of the claims, up to the first that reports a failure,
  // which is returned
  Failure collect() {
    std::lock_guard<std::mutex> lock(mu_);
    for (; tail_ < head_ && slots_[tail_ % kSlots].state == kFree; ++tail_) {}
    for (uint64_t at = head_ - tail_ > kSlots ? head_ - kSlots : tail_; at < head_; ++at) {
      Slot& s = slots_[at % kSlots];
      const int word = words_[at % kSlots];
      if (s.state != kLaunched || word == kPending) continue;
      s.state = kFree;
      if (word != 0) return Failure{word, s.what};
    }
    return Failure{0, nullptr};
  }
  // a bound for outstanding(): the calls made so far
  uint64_t now() {
    std::lock_guard<std::mutex> lock(mu_);
    return head_;
  }
  // device of a launched call from before `bound` whose word has not been collected; -1: there is none
  int outstanding(uint64_t bound) {
    std::lock_guard<std::mutex> lock(mu_);
    for (const Slot& s : slots_)
      if (s.state == kLaunched && s.at < bound) return s.device;
    return -1;
  }

 private:
  enum State { kFree, kClaimed, kLaunched };
  struct Slot {
    State state = kFree;
    int device = 0;
    const char* what = nullptr;
    uint64_t at = 0;
  };
  std::mutex mu_;
  volatile int* words_;
  Slot slots_[kSlots];
  uint64_t head_ = 0, tail_ = 0;   // claim number `at` takes slot at % kSlots; no slot in use has a number below tail_
};

}  // namespace fmb
