"""Bounds of the kernels' waits against one another, read from their source (running one out on a GPU would take seconds)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chatglm_cpp_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def _constant(name):
    return int(re.search(rf"constexpr unsigned long long {name} = (\d+)ull;", _source("common.cuh")).group(1))


def test_a_gate_runs_out_before_the_barriers_behind_it():
    """A launch of a host-buffer call waits for two words in turn, written by copies that may take their time; its other warps wait
    for what follows.  Theirs must be the longer bound, or they give up first and end the wait for the copies early."""
    assert _constant("kWaitLimitNs") > 2 * _constant("kGateLimitNs")
    gate = _source("decode_rope.cuh").split("bool wait_gate(")[1].split("\n}")[0]
    assert "kGateLimitNs" in gate


def test_the_loops_around_the_waits_outlast_their_clocks():
    """The polls of a gate are at least 200 ns apart on average, an attempt at a barrier suspends for up to 100 us but may return at
    once; the loop counts must not be what ends a wait early at those paces."""
    spins = 1 << int(re.search(r"constexpr unsigned int kSpinLimit = 1u << (\d+);", _source("common.cuh")).group(1))
    assert spins * 200 > _constant("kGateLimitNs")
    assert spins * 500 > _constant("kWaitLimitNs")   # half a microsecond: a failed attempt, two loads, the clock
