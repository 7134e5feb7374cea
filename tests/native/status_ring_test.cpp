// fmb::StatusRing with the GPU's stores made by the test; exits with the number of the check that failed.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

#include "../../flash_moba_b200/csrc/fmb_status_ring.h"

#define CHECK(n, cond)                                        \
  do {                                                        \
    if (!(cond)) {                                            \
      std::fprintf(stderr, "check %d: %s\n", n, #cond);       \
      std::exit(n);                                           \
    }                                                         \
  } while (0)

using fmb::StatusRing;

int main() {
  static volatile int words[StatusRing::kSlots];
  {  // a call that has claimed its slot but not been launched is neither passed over nor handed out again
    StatusRing r(words);
    const int a = r.claim("a", 0);
    std::thread other([&] {
      CHECK(1, r.collect().code == 0 && r.outstanding(r.now()) == -1);
      std::vector<int> rest;
      for (int i = 1; i < StatusRing::kSlots; ++i) {
        rest.push_back(r.claim("b", 1));
        CHECK(2, rest.back() >= 0 && rest.back() != a);
      }
      CHECK(3, r.claim("c", 1) == -1);
      for (int i : rest) { r.launched(i); *r.word(i) = 0; }
      CHECK(4, r.collect().code == 0 && r.outstanding(r.now()) == -1);
    });
    other.join();
    r.launched(a);
    CHECK(5, r.outstanding(r.now()) == 0 && r.collect().code == 0);
    *r.word(a) = 7;
    const StatusRing::Failure f = r.collect();
    CHECK(6, f.code == 7 && f.what[0] == 'a');
    CHECK(7, r.outstanding(r.now()) == -1 && r.collect().code == 0);
  }
  {  // a word that is late holds back no other; a withdrawn slot is free
    StatusRing r(words);
    const int late = r.claim("late", 0), bad = r.claim("bad", 0), none = r.claim("none", 0);
    r.launched(late);
    r.launched(bad);
    r.withdraw(none);
    *r.word(bad) = 3;
    CHECK(8, r.collect().code == 3);
    const uint64_t so_far = r.now();
    for (int i = 1; i < StatusRing::kSlots; ++i) {
      const int s = r.claim("x", 0);
      CHECK(9, s >= 0 && s != late);
      r.launched(s);
    }
    CHECK(10, r.claim("y", 0) == -1);
    *r.word(late) = 0;
    CHECK(11, r.collect().code == 0 && r.outstanding(so_far) == -1 && r.outstanding(r.now()) == 0);
  }
  {  // several threads: every failure is reported exactly once
    StatusRing r(words);
    std::atomic<int> sent{0}, got{0};
    auto take = [&] { while (r.collect().code != 0) ++got; };
    std::vector<std::thread> t;
    for (int id = 0; id < 4; ++id)
      t.emplace_back([&, id] {
        for (int i = 0; i < 20000; ++i) {
          int s;
          while ((s = r.claim("t", id)) < 0) take();
          if (i % 7 == 0) { r.withdraw(s); continue; }
          r.launched(s);
          const int code = i % 5 == 0 ? 4 : 0;
          sent += code != 0;
          *r.word(s) = code;
          if (i % 3 == 0) take();
        }
      });
    for (auto& x : t) x.join();
    take();
    CHECK(12, sent == got && r.outstanding(r.now()) == -1);
  }
  return 0;
}
