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
    bool fresh = false;
    // Launches in turn from three streams, and captures in between: more of each than there are slots.
    std::set<int> streams, graphs;
    int moved = 0, again = 0;
    for (int i = 0; i < 4 * kMeetingSlots; ++i) {
        const int slot = slots.of_stream(1 + i % 3);
        streams.insert(slot);
        moved += slot != slots.of_stream(1 + i % 3);
    }
    // A graph of 32 launches has one slot (two where it forks), every further graph its own.
    const int kGraphs = 40;
    for (int graph = 0; graph < kGraphs; ++graph)
        for (int launch = 0; launch < 32; ++launch) {
            const int slot = slots.of_capture(7 + graph, 1 + launch % 2, fresh);
            again += fresh != (launch < 2);
            graphs.insert(slot);
        }
    int shared = 0;
    for (int slot : graphs) shared += (int)streams.count(slot);
    printf("%d %d %d %d %d\\n", (int)streams.size(), moved, (int)graphs.size(), again, shared);

    // A slot that is given back goes to a later graph, once.
    const int returned = slots.of_capture(7, 1, fresh);
    slots.give_back(returned);
    slots.give_back(returned);
    const int next = slots.of_capture(1000, 1, fresh), other = slots.of_capture(1001, 1, fresh);
    printf("%d %d\\n", next == returned, (int)(graphs.count(other) + streams.count(other)));

    // Streams without end: all that find no slot share one that is nobody else's, and leave slots to captures.
    std::set<int> all;
    int outside = 0;
    for (int id = 100; id < 100 + 2 * kMeetingSlots; ++id) {
        const int slot = slots.of_stream(id);
        if (slot == kMeetingShared) { ++outside; continue; }
        all.insert(slot);
    }
    for (int id = 1; id <= 3; ++id) all.insert(slots.of_stream(id));
    const int late = slots.of_capture(5000, 1, fresh);
    printf("%d %d %d %d\\n", (int)all.size() == kMeetingStreams, outside == 2 * kMeetingSlots - kMeetingStreams + 3, late >= 0 && !all.count(late),
           slots.of_stream(100) != kMeetingShared);

    // Captures without end: refused when none is left, served again when one comes back.
    int kept = 0, slot = 0, last = -1;
    for (int capture = 10000; (slot = slots.of_capture(capture, 1, fresh)) >= 0; ++capture) { ++kept; last = slot; }
    const bool refused = slots.of_capture(50000, 1, fresh) < 0;
    slots.give_back(last);
    printf("%d %d %d\\n", kept <= kMeetingSlots, refused, slots.of_capture(50001, 1, fresh) == last);

    // From several threads.
    MeetingSlots fresh_slots;
    std::vector<std::thread> threads;
    std::vector<std::set<int>> found(8);
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            for (int i = 0; i < 2000; ++i) {
                bool is_new = false;
                found[t].insert(fresh_slots.of_stream(t));
                const int mine = fresh_slots.of_capture(100 * i + t, 0, is_new);
                if (mine < 0 || !is_new) found[t].insert(-1);
                fresh_slots.give_back(mine);
            }
        });
    for (auto& thread : threads) thread.join();
    std::set<int> together;
    int sum = 0;
    for (auto& mine : found) { sum += (int)mine.size(); together.insert(mine.begin(), mine.end()); }
    printf("%d %d %d\\n", sum, (int)together.size(), (int)together.count(-1));
    return 0;
}
"""


def test_launches_that_may_run_together_have_slots_of_their_own(tmp_path):
    steady, back, endless, captures, threads = host_program(tmp_path, PROGRAM)
    assert steady == (3, 0, 80, 0, 0)   # a slot per stream that stays; two per forked graph; none in common
    assert back == (1, 0)
    assert endless == (1, 1, 1, 1)
    assert captures == (1, 1, 1)
    assert threads == (8, 8, 0)
