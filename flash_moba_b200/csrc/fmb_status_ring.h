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
      const int i = (next_ + n) % kSlots;
      if (slots_[i].state != kFree) continue;
      next_ = (i + 1) % kSlots;
      words_[i] = kPending;
      slots_[i] = Slot{kClaimed, device, what, ++count_};
      return i;
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
  // frees the slots whose words have arrived, up to the first that reports a failure, which is returned
  Failure collect() {
    std::lock_guard<std::mutex> lock(mu_);
    for (int n = 0; n < kSlots; ++n) {
      const int i = (next_ + n) % kSlots;               // about the order of the claims
      if (slots_[i].state != kLaunched || words_[i] == kPending) continue;
      slots_[i].state = kFree;
      if (words_[i] != 0) return Failure{words_[i], slots_[i].what};
    }
    return Failure{0, nullptr};
  }
  // claims so far: what outstanding() is asked about
  uint64_t claims() {
    std::lock_guard<std::mutex> lock(mu_);
    return count_;
  }
  // device of a launched call among the first `claims` whose word has not been collected; -1: there is none
  int outstanding(uint64_t claims) {
    std::lock_guard<std::mutex> lock(mu_);
    for (const Slot& s : slots_)
      if (s.state == kLaunched && s.claim <= claims) return s.device;
    return -1;
  }

 private:
  enum State { kFree, kClaimed, kLaunched };
  struct Slot {
    State state = kFree;
    int device = 0;
    const char* what = nullptr;
    uint64_t claim = 0;
  };
  std::mutex mu_;
  volatile int* words_;
  Slot slots_[kSlots];
  int next_ = 0;
  uint64_t count_ = 0;
};

}  // namespace fmb
