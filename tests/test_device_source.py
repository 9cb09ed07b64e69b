"""Rules the device sources keep that no run can show to be broken reliably."""
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "opendba_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*", "", text)


def test_no_collective_over_the_lanes_that_happen_to_be_together():
    # __activemask() names the lanes that run together at the moment, not those
    # that will reach a shuffle
    for name in os.listdir(CSRC):
        if name.endswith((".cu", ".cuh")):
            assert "__activemask" not in _source(name), name


def test_feeder_decides_by_one_read():
    # the feeding warp's lanes take part in shuffles by what shared counters and
    # the timer say: one lane reads them for all
    text = _source("dtw_block.cuh")
    feeder = text[text.index("if (w == kBlkWarps) {"):text.index("if (w >= wact) return false;")]
    assert "warp_count(" in feeder and "warp_timer_ns(" in feeder
    assert "smem_count(" not in feeder and "global_timer_ns(" not in feeder


def test_lanes_read_what_lane_0_acquired_after_a_warp_barrier():
    text = _source("dtw_block.cuh")
    staged = text[text.index("gate.ready("):text.index("__ldcg(job.edge_in")]
    assert "__syncwarp()" in staged
    text = _source("dtw_warp.cuh")
    assert "__syncwarp()" in text[text.index("gate.wait("):text.index("__ldcg(")]


def test_waits_of_the_sweep_take_the_launch_limit():
    # the limit a launch (or the self-test) gives is the one its sweep's waits
    # run out by, and there is no second wait beside them to test instead
    text = _source("dtw_block.cuh")
    assert "gate.limit()" in text and "kWaitLimitNs" not in text
    assert "wait_in" not in _source("dtw_pipe.cuh")
    pairs = _source("dtw_pairwise.cu")
    kernel = pairs[pairs.index("gate_selftest_kernel(SelfTest"):]
    assert "sweep_block<" in kernel[:kernel.index("int gate_selftest(")]


def test_every_sweep_has_an_error_word():
    # a wait that runs out without one would leave a wrong result unsaid
    for name in ("dba_round.cu", "dtw_pairwise.cu"):
        assert "NoGate()" not in _source(name), name
    assert "return nullptr" not in _source("dtw_device.cuh")


def test_large_scratch_is_not_mapped_through_the_pool():
    # mapping and unmapping 100 GB through a pool takes two seconds, a plain
    # allocation a sixtieth of one
    text = _source("capi.cu")
    alloc = text[text.index("cudaError_t scratch_alloc("):text.index("int scratch_trim()")]
    assert "bytes > kScratchKeepBytes) return cudaMalloc(" in alloc
    assert "cudaFree(p)" in alloc
