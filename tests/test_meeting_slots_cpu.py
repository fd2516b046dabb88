"""The meeting slots of the single-launch MLP: launches that may run at the same time never get the same one."""

from tests.helpers import host_program

PROGRAM = """
#include <cstdio>
#include <set>
#include <thread>
#include <vector>
#include "meeting_slots.h"
using namespace mt;
int main() {
    MeetingSlots slots;
    // Launches in turn from three streams, more than there are slots.
    std::set<int> streams, graphs;
    int moved = 0;
    for (int i = 0; i < 2 * kMeetingSlots; ++i) {
        const int slot = slots.of_stream(1 + i % 3);
        streams.insert(slot);
        moved += slot != slots.of_stream(1 + i % 3);
    }
    // A graph of 32 launches has one slot (two where it forks), every further graph its own.
    for (int graph = 0; graph < 40; ++graph)
        for (int launch = 0; launch < 32; ++launch) graphs.insert(slots.of_capture(7 + graph, 1 + launch % 2));
    int shared = 0;
    for (int slot : graphs) shared += (int)streams.count(slot);
    printf("%d %d %d %d\\n", (int)streams.size(), moved, (int)graphs.size(), shared);

    // Streams without end: all that find no slot share one that is nobody else's, and leave slots to captures.
    std::set<int> all = graphs;
    int outside = 0;
    for (int id = 100; id < 100 + 2 * kMeetingStreams; ++id) {
        const int slot = slots.of_stream(id);
        if (slot == kMeetingShared) ++outside;
        else all.insert(slot);
    }
    for (int id = 1; id <= 3; ++id) all.insert(slots.of_stream(id));
    printf("%d %d %d\\n", (int)all.size() == kMeetingStreams + 80, outside == kMeetingStreams + 3, slots.of_stream(100) != kMeetingShared);

    // Captures without end: each has a slot of its own until none is left, and those keep theirs.
    int slot = 0, capture = 10000;
    for (; (slot = slots.of_capture(capture, 1)) >= 0; ++capture) all.insert(slot);
    printf("%d %d %d %d\\n", (int)all.size() == kMeetingSlots, capture - 10000 == kMeetingSlots - kMeetingStreams - 80, slots.of_capture(capture + 1, 1),
           slots.of_capture(capture - 1, 1) == kMeetingSlots - 1);

    // From several threads.
    MeetingSlots others;
    std::vector<std::thread> threads;
    std::vector<std::set<int>> found(8);
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            for (int i = 0; i < 2000; ++i) {
                found[t].insert(others.of_stream(t));
                found[t].insert(others.of_capture(i, t));
            }
        });
    for (auto& thread : threads) thread.join();
    std::set<int> together;
    int sum = 0;
    for (auto& mine : found) { sum += (int)mine.size(); together.insert(mine.begin(), mine.end()); }
    printf("%d %d %d\\n", sum, (int)together.size(), *together.begin());
    return 0;
}
"""


def test_launches_that_may_run_together_have_slots_of_their_own(tmp_path):
    steady, endless, captures, threads = host_program(tmp_path, PROGRAM)
    assert steady == (3, 0, 80, 0)   # a slot per stream that stays; two per forked graph; none in common
    assert endless == (1, 1, 1)
    assert captures == (1, 1, -1, 1)
    assert threads == (8 * 2001, 8 * 2001, 0)
