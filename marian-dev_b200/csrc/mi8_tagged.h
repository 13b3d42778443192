// The host's wait for words that a kernel writes to pinned memory, each with a tag in its upper half that says it is new.  No CUDA in here.
#pragma once

namespace mi8 {

enum class TaggedWait { kArrived, kMissing, kFailed };
enum class StreamState { kBusy, kIdle, kFailed };

// Until words[0..n) all carry `tag`.  `pause` is called between looks; every `turns` of them `state` says what the stream does that the words come from: once it
// is idle all that its kernels wrote is here, so that a word which still has another tag will not come (a launch that failed or gave up never writes it).
template <typename Pause, typename State>
TaggedWait wait_for_tagged(const volatile unsigned long long* words, int n, unsigned tag, unsigned turns, Pause&& pause, State&& state) {
  const auto arrived = [&](int i) { return static_cast<unsigned>(words[i] >> 32) == tag; };
  int i = 0;
  for(unsigned turn = 1;; ++turn) {
    while(i < n && arrived(i))
      ++i;
    if(i == n)
      return TaggedWait::kArrived;
    pause();
    if(turn % turns == 0) {
      const StreamState s = state();
      if(s == StreamState::kFailed)
        return TaggedWait::kFailed;
      if(s == StreamState::kIdle && !arrived(i))   // (looked at once more: it may have come before the stream was asked)
        return TaggedWait::kMissing;
    }
  }
}

}  // namespace mi8
