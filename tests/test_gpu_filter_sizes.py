"""The frequency filter at the lengths where its transform changes: the
shortest traces, both sides of a power of two, 16 points a thread, and the
first length that takes the cuFFT form.  The bar is the filter's: rel-L2 of
the filtered traces against the oracle's float64 restatement <= 1e-4, traces
of zeros untouched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt", [5, 64, 256, 257, 2048, 2049, 4096, 8192, 8193, 16384, 16385])
def test_filter_lengths_match_oracle(engine, oracle, nt):
    rng = np.random.default_rng(nt)
    x = np.cumsum(rng.standard_normal((5, nt)), axis=1).astype(np.float32)
    x[2] = 0.0
    got = engine.freq_filter(x, 2e-3, 3, 5.0, 40.0)
    want = oracle.freq_filter(x, 2e-3, 3, 5.0, 40.0)
    assert np.linalg.norm(want) > 0
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 1e-4
    assert np.array_equal(got[2], x[2])
