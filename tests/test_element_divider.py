"""The multiply-and-shift division by which the stage kernels find an element's place in a
box (nwb::set_divider), restated here and compared with integer division over its range."""
import numpy as np
import pytest


def divider(d):
    L = 0
    while (1 << L) < d:
        L += 1
    shift = 25 + L
    return ((1 << shift) + d - 1) // d, shift


@pytest.mark.parametrize("seed", [0, 1])
def test_quotients_are_exact_below_2_to_25(seed):
    rng = np.random.default_rng(seed)
    ds = list(range(1, 600)) + [int(x) for x in rng.integers(1, (1 << 25) + 1, 400)] + [1 << 25, (1 << 25) - 1]
    for d in ds:
        mul, shift = divider(d)
        assert mul < 1 << 32
        q = rng.integers(0, (1 << 25) // d + 1, 40)
        n = np.concatenate([q * d, q * d - 1, rng.integers(0, 1 << 25, 40), [0, (1 << 25) - 1]])
        n = np.unique(n[(n >= 0) & (n < 1 << 25)])
        assert [(int(x) * mul) >> shift for x in n] == [int(x) // d for x in n], d
