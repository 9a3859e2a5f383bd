"""The rule by which blocks of an on-chip elastic shot leave after a wait that ran
out (csrc/halo_exit.cuh), on the CPU: no block may leave while edge rows are on
their way to it.

Two neighbouring blocks X and Y at the end of a launch.  X sends, waits, and gives
up at its limit; Y runs late.  Y's rows take a flight time to arrive; Y's own wait
succeeds at once, since X sent before it waited.  Times in nanoseconds."""
import itertools
import os
import subprocess

import hmclab_gb300 as H

_SOURCE = r"""
#include "halo_exit.cuh"
#include <cstdio>
#include <cstdlib>
int main(int argc, char** argv) {
  printf("%llu %d %d %d %d\n", hmc::fwi::HALO_DRAIN_NS, hmc::fwi::halo_must_drain(false, 0), hmc::fwi::halo_must_drain(false, 1),
         hmc::fwi::halo_must_drain(true, 0), hmc::fwi::halo_must_drain(true, 1));
}
"""


def _rule(tmp_path):
    src, exe = tmp_path / "e.cpp", tmp_path / "e"
    src.write_text(_SOURCE)
    csrc = os.path.join(os.path.dirname(H.__file__), "csrc")
    subprocess.run(["g++", "-std=c++17", "-I", csrc, str(src), "-o", str(exe)], check=True)
    ns, *must = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    return ns, lambda gave_up, status: bool(must[2 * int(gave_up) + int(status)])


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
    drain_ns, must_drain = _rule(tmp_path)
    assert _violations(drain_ns, must_drain) == 0
    assert not must_drain(False, False)  # no cost where nothing ran out
    # the check sees a rule in which only the receiver that gave up stays
    assert _violations(drain_ns, lambda gave_up, status: gave_up) > 0
