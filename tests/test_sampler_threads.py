"""The threads that build rows ahead of the accept loop: one crew for all samplers, its limit kept at any time, given back when idle,
absent in a forked child."""
import os
import sys
import time

import numpy as np
import pytest

from dflb import pkg


def _threads():
    return len(os.listdir("/proc/self/task"))


def _block(vocab, seed=1):
    rng = np.random.default_rng(seed)
    rows = (rng.standard_normal((16, vocab)) * 2).astype(np.float32)
    favourite = rng.integers(0, vocab, 16)
    rows[np.arange(16), favourite] = 40.0
    return rows, [0] + [int(f) for f in favourite[:15]]


def test_samplers_share_their_threads_and_give_them_back():
    before = _threads()
    rows, block = _block(20000)
    samplers = [pkg.Sampler(temperature=0.7, top_p=0.95, seed=i) for i in range(16)]
    for s in samplers:
        assert len(pkg.accept_prefix(block, rows, 20000, None, s, 100, ())["accepted_drafts"]) == 15
    assert _threads() - before <= max(2, os.cpu_count())
    deadline = time.monotonic() + 20
    while _threads() > before and time.monotonic() < deadline:
        time.sleep(0.1)
    assert _threads() <= before      # with every sampler still there
    assert len(pkg.accept_prefix(block, rows, 20000, None, samplers[0], 100, ())["accepted_drafts"]) == 15


@pytest.mark.skipif(len(os.sched_getaffinity(0)) < 4, reason="needs four cores to tell two workers from more")
def test_a_limit_set_after_the_first_block_holds():
    rows, block = _block(151936)
    s = pkg.Sampler(temperature=1.0, seed=3)     # no top-p: a row is ordered, milliseconds of work each
    decide = lambda: pkg.accept_prefix(block, rows, 151936, None, s, 100, ())
    decide()
    s.set_worker_threads(2)
    cpu, wall = time.process_time(), time.perf_counter()
    for _ in range(3):
        decide()
    cpu, wall = time.process_time() - cpu, time.perf_counter() - wall
    assert cpu < 2.4 * wall      # two at work at a time


def test_a_forked_child_decides_blocks_and_ends():
    rows, block = _block(20000)
    s = pkg.Sampler(temperature=0.7, top_p=0.95, seed=3)
    pkg.accept_prefix(block, rows, 20000, None, s, 100, ())
    sys.stdout.flush()
    child = os.fork()
    if child == 0:
        code = 1
        try:
            code = 0 if len(pkg.accept_prefix(block, rows, 20000, None, s, 100, ())["accepted_drafts"]) == 15 else 2
            s.close()
        finally:
            os._exit(code)
    deadline = time.monotonic() + 60
    while time.monotonic() < deadline:
        pid, status = os.waitpid(child, os.WNOHANG)
        if pid:
            assert os.waitstatus_to_exitcode(status) == 0
            return
        time.sleep(0.02)
    os.kill(child, 9)
    os.waitpid(child, 0)
    raise AssertionError("the child did not end")
