// Which launches share the memory in which the CTAs of a single-launch MLP meet (a counter and a flag per CTA, in
// affine_mlp_fused.cuh).  Two launches that may run at the same time must not: each would count the other's arrivals.
//
// A slot is safe where the call's workspace is.  Launches of one stream run in order, and a launch touches its slot behind
// its wait for the kernel in front, so a stream has one slot.  A captured launch runs whenever its graph is replayed,
// beside any stream and any other graph, but in order with what the same stream captured in the same sequence: those
// share a slot that nothing else is ever given.  (To learn that a graph is gone takes an object that the graph retains, and with
// one a replay takes 2 us longer and its launch 8 us of the host's time; slots are small instead, and many.)
#pragma once

#include <map>
#include <mutex>
#include <utility>

namespace mt {

constexpr int kMeetingSlots = 16384;               // 1 MB; with 2 MB a program's buffers come to lie elsewhere, and decode attention of 16 x
                                                   // 2048 tokens, which has nothing to do with it, takes 12.46 us instead of 12.32
constexpr int kMeetingStreams = 512;               // slots that streams may take; they are not told when a stream ends
constexpr int kMeetingShared = kMeetingSlots;      // of all later streams, whose launches the caller puts in one order
constexpr int kMeetingSelfTest = kMeetingSlots + 1;
constexpr int kMeetingSlotsInAll = kMeetingSlots + 2;

class MeetingSlots {
public:
    // The slot of a stream, by its id (not its handle, which another stream may get later); kMeetingShared when all are taken.
    int of_stream(unsigned long long stream) {
        const std::lock_guard<std::mutex> lock(mutex_);
        const auto found = streams_.find(stream);
        if (found != streams_.end()) return found->second;
        if ((int)streams_.size() == kMeetingStreams || next_ == kMeetingSlots) return kMeetingShared;
        streams_.emplace(stream, next_);
        return next_++;
    }

    // The slot of what `stream` (a name that is its own while it captures) captures in the sequence `capture`; -1 when all
    // are taken.
    int of_capture(unsigned long long capture, unsigned long long stream) {
        const std::lock_guard<std::mutex> lock(mutex_);
        const std::pair<unsigned long long, unsigned long long> key(capture, stream);
        const auto found = captures_.find(key);
        if (found != captures_.end()) return found->second;
        if (next_ == kMeetingSlots) return -1;
        captures_.emplace(key, next_);
        return next_++;
    }

private:
    std::mutex mutex_;
    std::map<unsigned long long, int> streams_;
    std::map<std::pair<unsigned long long, unsigned long long>, int> captures_;
    int next_ = 0;
};

}  // namespace mt
