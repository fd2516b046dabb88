// Which launches share the memory in which the CTAs of a single-launch MLP meet (a counter and a flag per CTA, in
// affine_mlp_fused.cuh).  Two launches that may run at the same time must not: each would count the other's arrivals.
//
// A slot is safe where the call's workspace is.  Launches of one stream run in order, and a launch touches its slot behind
// its wait for the kernel in front, so a stream has one slot.  A captured launch runs whenever its graph is replayed,
// beside any stream and any other graph, but in order with what the same stream captured in the same sequence: those
// share a slot that nothing else gets while the graph lives.
//
// Host code without CUDA calls: the lock is never held across one, so a graph's destructor may give a slot back at any time.
#pragma once

#include <map>
#include <mutex>
#include <utility>
#include <vector>

namespace mt {

constexpr int kMeetingSlots = 1024;
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
        if ((int)streams_.size() == kMeetingStreams) return kMeetingShared;
        const int slot = take();
        if (slot < 0) return kMeetingShared;
        streams_.emplace(stream, slot);
        return slot;
    }

    // The slot of what `stream` (a name that is its own while it captures) captures in the sequence `capture`; -1 when all
    // are taken.  `fresh`: the caller has to see to it that give_back() is called when the graph and all that was made
    // of it are gone.
    int of_capture(unsigned long long capture, unsigned long long stream, bool& fresh) {
        const std::lock_guard<std::mutex> lock(mutex_);
        const std::pair<unsigned long long, unsigned long long> key(capture, stream);
        const auto found = captures_.find(key);
        fresh = found == captures_.end();
        if (!fresh) return found->second;
        const int slot = take();
        if (slot >= 0) captures_.emplace(key, slot);
        return slot;
    }

    void give_back(int slot) {
        const std::lock_guard<std::mutex> lock(mutex_);
        for (auto it = captures_.begin(); it != captures_.end(); ++it) {
            if (it->second != slot) continue;
            captures_.erase(it);
            free_.push_back(slot);
            return;
        }
    }

private:
    int take() {
        if (!free_.empty()) {
            const int slot = free_.back();
            free_.pop_back();
            return slot;
        }
        return next_ < kMeetingSlots ? next_++ : -1;
    }

    std::mutex mutex_;
    std::map<unsigned long long, int> streams_;
    std::map<std::pair<unsigned long long, unsigned long long>, int> captures_;
    std::vector<int> free_;
    int next_ = 0;
};

}  // namespace mt
