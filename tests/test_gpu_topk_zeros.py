"""Top-k whose threshold is zero: the reference compares values, so -0 and 0 are ties, and all of them are kept.  The draws lie in the
middle of the intervals of tokens at -0, which a threshold compared by its bits would drop."""
import numpy as np
import pytest

from tests.test_gpu_sampling import dev, pool  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [777, 4096])
@pytest.mark.parametrize("zeros,top_k", [(30, 15), (300, 200)])   # finished on a list, and pass by pass
@pytest.mark.parametrize("temperature", [1.0, 0.8])
def test_zeros_of_both_signs_are_ties(pool, oracle, V, zeros, top_k, temperature):  # noqa: F811
    rng = np.random.default_rng(V + zeros)
    row = (-1.0 - rng.random(V)).astype(np.float32)
    at = rng.permutation(V)[:10 + zeros]
    row[at[:10]] = 1.0 + rng.random(10)
    row[at[10:]] = np.where(np.arange(zeros) % 2, np.float32(-0.0), np.float32(0.0))
    cfg = oracle.sampler_cfg(temperature=temperature, top_k=top_k)
    _, probs = oracle.sampler_sample(cfg, row, 0.5, return_probs=True)
    cum = np.cumsum(probs.astype(np.float64))
    want = np.sort(at[11::2])[:12]
    assert np.signbit(row[want]).all() and (probs > 0).sum() == 10 + zeros
    draws = (cum[want] - probs[want] / 2).astype(np.float32)
    got = pool.sample(np.tile(row, (len(want), 1)), draws, temperature=temperature, top_k=top_k)
    assert got.tolist() == want.tolist()
