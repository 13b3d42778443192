// wait_for_tagged on the CPU: a thread in the place of the GPU writes the words, in any order, late, in part or not at all.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>

#include "../../marian-dev_b200/csrc/mi8_tagged.h"

using namespace mi8;

namespace {
int failures = 0;
void expect(bool ok, const char* what) {
  if(!ok) {
    std::printf("failed: %s\n", what);
    ++failures;
  }
}
unsigned long long word(unsigned tag, unsigned value) { return static_cast<unsigned long long>(tag) << 32 | value; }
}  // namespace

int main() {
  const int n = 6;
  const auto nothing = []() {};
  const auto idle = []() { return StreamState::kIdle; };
  {
    std::vector<unsigned long long> w(n, word(7, 1));
    expect(wait_for_tagged(w.data(), n, 7u, 1u, nothing, idle) == TaggedWait::kArrived, "all there");
    expect(wait_for_tagged(w.data(), 0, 8u, 1u, nothing, idle) == TaggedWait::kArrived, "no words");
  }
  // an idle stream and one word that is missing, whichever it is and whatever the others carry
  for(int missing = 0; missing < n; ++missing)
    for(unsigned old : {0u, 6u}) {
      std::vector<unsigned long long> w(n, word(7, 1));
      w[missing] = word(old, 1);
      int asked = 0;
      const auto state = [&]() { return ++asked < 5 ? StreamState::kBusy : StreamState::kIdle; };
      expect(wait_for_tagged(w.data(), n, 7u, 3u, nothing, state) == TaggedWait::kMissing && asked == 5, "one word missing");
    }
  // a word that comes between the last look and the answer that the stream is idle
  for(int late = 0; late < n; ++late) {
    std::vector<unsigned long long> w(n, word(7, 1));
    w[late] = 0;
    const auto state = [&]() {
      w[late] = word(7, 2);
      return StreamState::kIdle;
    };
    expect(wait_for_tagged(w.data(), n, 7u, 1u, nothing, state) == TaggedWait::kArrived, "a word that comes late");
  }
  {
    std::vector<unsigned long long> w(n, 0ull);
    expect(wait_for_tagged(w.data(), n, 7u, 1u, nothing, []() { return StreamState::kFailed; }) == TaggedWait::kFailed, "a stream that failed");
  }
  // another thread writes them one by one, last first
  for(int round = 1; round <= 20; ++round) {
    std::vector<unsigned long long> w(n, word(round - 1, 0));
    std::atomic<bool> done{false};
    std::thread writer([&]() {
      for(int i = n - 1; i >= 0; --i) {
        std::this_thread::sleep_for(std::chrono::microseconds(200));
        reinterpret_cast<std::atomic<unsigned long long>*>(w.data())[i].store(word(round, i));
      }
      done = true;
    });
    const auto state = [&]() { return done ? StreamState::kIdle : StreamState::kBusy; };
    const bool ok = wait_for_tagged(w.data(), n, static_cast<unsigned>(round), 16u, []() { std::this_thread::yield(); }, state) == TaggedWait::kArrived;
    writer.join();
    expect(ok && w[0] == word(round, 0) && w[n - 1] == word(round, n - 1), "words of another thread");
  }
  if(failures == 0)
    std::printf("tagged wait tests passed\n");
  return failures;
}
