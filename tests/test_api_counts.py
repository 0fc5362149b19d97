"""Counts that the Python calls take: what is no whole number is a TypeError."""
import numpy as np
import pytest


@pytest.mark.parametrize("n", [2.0, "2", np.float64(2)])
def test_counts_that_are_no_whole_numbers(lib, n):
    import mrg8_gb300 as m
    g = m.MRG8(1)
    out = np.zeros(4)
    with pytest.raises(TypeError):
        g.rand(out, n)
    with pytest.raises(TypeError):
        g.randint(np.zeros(4, dtype=np.uint32), n)
    assert not out.any()
