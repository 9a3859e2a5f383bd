"""The rules by which the blocks of an on-chip elastic shot exchange edge rows
(csrc/halo_rules.cuh), on the CPU: no block may leave while rows are on their way
to it, and no lane may wait for a phase that the barrier can leave behind.

Leaving: two neighbouring blocks X and Y at the end of a launch.  X sends, waits,
and gives up at its limit; Y runs late.  Y's rows take a flight time to arrive; Y's
own wait succeeds at once, since X sent before it waited.  Times in nanoseconds."""
import itertools
import os
import subprocess

import hmclab_gb300 as H

_SOURCE = r"""
#include "halo_rules.cuh"
#include <cstdio>
#include <cstdlib>
int main(int argc, char** argv) {
  using namespace hmc::fwi;
  printf("%llu %d %d %d %d %d %d %d %d\n", HALO_DRAIN_NS, halo_must_drain(false, 0), halo_must_drain(false, 1),
         halo_must_drain(true, 0), halo_must_drain(true, 1), halo_sends(false), halo_sends(true), halo_awaits(false),
         halo_awaits(true));
}
"""


def _rule(tmp_path):
    src, exe = tmp_path / "e.cpp", tmp_path / "e"
    src.write_text(_SOURCE)
    csrc = os.path.join(os.path.dirname(H.__file__), "csrc")
    subprocess.run(["g++", "-std=c++17", "-I", csrc, str(src), "-o", str(exe)], check=True)
    ns, *v = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    return ns, lambda gave_up, status: bool(v[2 * int(gave_up) + int(status)]), v[4:6], v[6:8]


def _leave(drain_ns, must_drain, limit, late, flight, step):
    """(time the blocks leave, time Y's rows have arrived at X)."""
    arrived = late + flight
    gave_up = arrived > limit
    end_x = limit if gave_up else arrived
    if must_drain(gave_up, gave_up):
        end_x += drain_ns
    read = late + step  # Y's read of the status word, after its last send
    end_y = read + (drain_ns if must_drain(False, gave_up and read >= limit) else 0)
    return max(end_x, end_y), arrived


def _violations(drain_ns, must_drain):
    bad = 0
    for limit, flight, step in itertools.product((1_000, 1_000_000), (1, 500, 5_000, 15_000), (1, 50, 2_000)):
        lates = [0, limit // 2] + [limit + k for k in range(-20_000, 100_000, 250)]
        for late in (t for t in lates if t >= 0):
            leave, arrived = _leave(drain_ns, must_drain, limit, late, flight, step)
            bad += leave < arrived
    return bad


def test_no_block_leaves_before_its_rows_arrived(tmp_path):
    drain_ns, must_drain, _, _ = _rule(tmp_path)
    assert _violations(drain_ns, must_drain) == 0
    assert not must_drain(False, False)  # no cost where nothing ran out
    # the check sees a rule in which only the receiver that gave up stays
    assert _violations(drain_ns, lambda gave_up, status: gave_up) > 0


def _stuck(lanes, steps=4):
    """Whether some order of events leaves a thread waiting for good.  `lanes`:
    (sends, waits) of the block's threads, the first of which arms the barrier.  Per
    step a thread waits for phase n (by parity, as the barrier is asked), the first
    arms it again, it sends, and all meet at the block's barrier; the neighbour
    completes phase n + 1 once it has every sender's rows of step n and the barrier is
    armed.  Phase 0 is complete at the start."""
    start = (tuple((0, 0) for _ in lanes), 1, 0)  # (step, stage) per thread, phases completed, arms beyond the first
    seen, todo = {start}, [start]
    while todo:
        threads, phases, arms = todo.pop()
        after = []
        for k, ((step, stage), (sends, waits)) in enumerate(zip(threads, lanes)):
            if step == steps:
                continue
            if stage == 0 and (not waits or phases % 2 != step % 2):
                after.append((k, (step, 1), phases, arms + (k == 0)))
            elif stage == 1:
                after.append((k, (step, 2), phases, arms))  # sent, if it sends
            elif stage == 2 and all(t >= (step, 2) for t in threads):
                after.append((k, (step + 1, 0), phases, arms))
        new = [(tuple(s if j == k else t for j, t in enumerate(threads)), p, a) for k, s, p, a in after]
        if all(t >= (phases - 1, 2) for t, (sends, _) in zip(threads, lanes) if sends) and arms >= phases:
            new.append((threads, phases + 1, arms))
        if not new and any(t[0] < steps for t in threads):
            return True
        for n in new:
            if n not in seen and n[1] <= steps + 2:
                seen.add(n)
                todo.append(n)
    return False


def test_no_lane_waits_for_a_phase_left_behind(tmp_path):
    _, _, sends, awaits = _rule(tmp_path)
    column, past = (bool(sends[1]), bool(awaits[1])), (bool(sends[0]), bool(awaits[0]))
    assert column == (True, True)
    assert not _stuck([column, column]) and not _stuck([column, past, column])
    # the check sees a lane that waits without sending
    assert _stuck([column, (False, True)])
