"""The nucleus without ordering the row against the ordered path (a registered row order selects it): same tokens, same draws."""
import importlib

import numpy as np
import pytest

pkg = importlib.import_module("qwen-llm_b200")


@pytest.mark.parametrize("vocab", [1023, 1024, 1025, 5003, 40007])
@pytest.mark.parametrize("shape", ["broad", "peaked", "ties", "constant", "half_masked", "offset"])
def test_nucleus_equals_ordered_path(vocab, shape):
    g = np.random.default_rng(vocab)
    x = (g.standard_normal((1, vocab)) * 2).astype(np.float32)
    if shape == "peaked":
        x[0, g.integers(0, vocab, 20)] += 15
    elif shape == "ties":
        x = np.round(x * 2) / 2 + 0.0   # one zero: the order of -0 and 0 is the f32 total order's
    elif shape == "constant":
        x[:] = -1.5
    elif shape == "half_masked":
        x[0, ::2] = -np.inf
    elif shape == "offset":
        x += 30000
    x = np.ascontiguousarray(x, dtype=np.float32)
    order = np.argsort(-x, axis=1, kind="stable").astype(np.uint32)
    for top_p, temperature in ((0.01, 1.0), (0.5, 0.3), (0.95, 0.7), (0.95, 2.0), (0.9999999, 1.0)):
        a = pkg.Sampler(temperature=temperature, top_p=top_p, seed=7)
        b = pkg.Sampler(temperature=temperature, top_p=top_p, seed=7)
        b.set_row_order(x, order)
        for _ in range(20):
            assert a.sample(x[0]) == b.sample(x[0])
        assert b.preordered_rows == 20 and a.preordered_rows == 0
        assert a.rng_state() == b.rng_state()
