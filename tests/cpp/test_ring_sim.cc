// The ring's flag protocol on host threads (sim/ring_sim.h) as its kernel runs it: the lanes of a group with
// their barrier, two groups that take the slices in turn and hand the order of their posts over, early credits
// of one group, several calls in a row. Run under ThreadSanitizer it also checks that every access to a FIFO
// slot is ordered by a counter. (The schedule itself: tests/test_cpu_ring_sim.py.)
#include "check.h"
#include "sim/ring_sim.h"

using namespace b200ccl;
using namespace b200ccl::sim;

int main() {
    for (Collective coll : {Collective::AllReduce, Collective::ReduceScatter, Collective::AllGather}) {
        for (int groups : {1, 2}) {
            for (int n : {2, 3}) {
                RingSimConfig c;
                c.nranks = n;
                c.channels = 2;
                c.collective = coll;
                c.redop = n == 2 ? RedOp::Avg : RedOp::Sum;
                c.groups = groups;
                c.lanes = 4;
                c.calls = 3;
                c.fifo_bytes = 4096;  // four slots of 256 floats: wraps many times
                c.count = 3001;
                for (int slow : {-1, 0, groups - 1}) {
                    c.slow_group = slow;
                    c.slow_rank = slow == 0 ? n - 1 : -1;
                    const RingSimResult r = run_ring_sim(c);
                    T_CHECK(r.wrong == 0 && !r.timed_out && r.slices > 0);
                }
                if (groups == 1) {  // slices small enough for an early credit, and both kinds in one message
                    c.slow_group = 0;
                    for (std::size_t early : {static_cast<std::size_t>(128), static_cast<std::size_t>(256)}) {
                        c.early_credit_elems = early;
                        const RingSimResult r = run_ring_sim(c);
                        T_CHECK(r.wrong == 0 && !r.timed_out);
                    }
                }
            }
        }
    }
    for (std::size_t count : {1, 5, 129, 1024}) {  // slices that are empty for one group or for both
        RingSimConfig c;
        c.nranks = 4;
        c.channels = 2;
        c.groups = 2;
        c.lanes = 2;
        c.calls = 4;
        c.count = count;
        const RingSimResult r = run_ring_sim(c);
        T_CHECK(r.wrong == 0 && !r.timed_out);
    }
    {   // the same slices as one group of one lane, whatever the split of the work
        RingSimConfig c;
        c.count = 20000;
        c.fifo_bytes = 16384;
        const RingSimResult one = run_ring_sim(c);
        c.groups = 2;
        c.lanes = 4;
        c.channels = 4;
        const RingSimResult two = run_ring_sim(c);
        T_CHECK(one.wrong == 0 && two.wrong == 0 && one.slices == two.slices && one.empty_slices == two.empty_slices);
    }
    {   // a rank that stops: its neighbours' bounded waits run out, both groups of everyone leave
        RingSimConfig c;
        c.channels = 1;
        c.groups = 2;
        c.lanes = 4;
        c.count = 1u << 14;
        c.fifo_bytes = 4096;
        c.stall_rank = 2;
        c.stall_after_slices = 3;
        c.wait_timeout_ms = 200.0;
        const RingSimResult r = run_ring_sim(c);
        T_CHECK(r.timed_out && r.timeout_rank != 2);
    }
#if !defined(__SANITIZE_THREAD__)  // a race by design
    {   // groups that do not wait for their turn publish slices that the slow one is still moving
        RingSimConfig c;
        c.channels = 1;
        c.groups = 2;
        c.count = 1u << 14;
        c.fifo_bytes = 4096;
        c.slow_group = 0;
        c.slow_rank = 0;
        c.wait_timeout_ms = 500.0;
        c.skip_turns = true;
        const RingSimResult r = run_ring_sim(c);
        T_CHECK(r.wrong != 0 || r.timed_out);
    }
#endif
    {   // bad configurations are refused
        RingSimConfig c;
        c.groups = 3;
        T_CHECK(run_ring_sim(c).wrong == -1);
        c.groups = 2;
        c.lanes = 5;
        T_CHECK(run_ring_sim(c).wrong == -1);
    }
    std::printf("ring sim ok\n");
    return 0;
}
