"""Row argmax and runner-up gap at the edges of its split of a row, and the two-matrix step's error word."""
import importlib

import numpy as np
import pytest

pkg = importlib.import_module("qwen-llm_b200")


def _expected(x):
    am = np.array([int(np.nonzero(np.isnan(r))[0][0]) ^ -1 if np.isnan(r).any() else int(np.argmax(r)) for r in x], np.int32)
    gap = []
    for r, a in zip(x, am):
        if a < 0 or r.size == 1:
            gap.append(0.0)
        else:
            gap.append(np.float32(r[a]) - np.delete(r, a).max())
    return am, np.array(gap, np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 16, 17])
@pytest.mark.parametrize("vocab", [1, 2, 7, 8, 9, 8191, 8193, 65535, 65537, 151936])
def test_argmax_of_a_split_row(rows, vocab):
    g = np.random.default_rng(rows * 1000003 + vocab)
    x = g.standard_normal((rows, vocab)).astype(np.float32)
    x[rows - 1] = np.round(x[rows - 1]) + 0.0        # ties: the lowest index wins
    x[0, vocab - 1] = 9.0                            # the last column of the last part
    if rows > 2 and vocab > 8:
        x[1, [vocab // 2, vocab - 2]] = np.nan       # reported, the first one
    am, gap = pkg.argmax_top2(x)
    want_am, want_gap = _expected(x)
    assert np.array_equal(am, want_am)
    assert np.array_equal(gap, want_gap)


@pytest.mark.gpu
def test_two_matrix_step_reports_overflow_and_recovers():
    ms = []
    for n_in, n_out in ((256, 256), (256, 512)):
        _, _, _, ptr, n_bytes = pkg.synth_tensor("w", pkg.Q4_K, n_in, n_out, 3 + n_out, 0.02)
        ms.append(pkg.QMatrix(pkg.Q4_K, n_in, n_out, pkg.device_to_host(ptr, n_bytes)))
        pkg.device_free(ptr)
    pipe = pkg.C1Pipeline(*ms)
    x = np.random.default_rng(0).standard_normal((5, 256)).astype(np.float32)
    am, gap, _, logits = pipe.step(x, np.zeros(5, np.int32), want_logits=True)
    assert np.array_equal(am, logits.argmax(1))
    with pytest.raises(pkg.DflError):
        pipe.step(x * 1e7, np.zeros(5, np.int32))    # outside the range of the f16 operands
    am2, gap2, _, _ = pipe.step(x, np.zeros(5, np.int32))
    assert np.array_equal(am, am2) and np.array_equal(gap, gap2)
    pipe.close()
