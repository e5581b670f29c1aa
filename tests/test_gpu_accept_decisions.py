"""Accept decisions close to their boundary: the draws lie 0.4 % of the acceptance probability to either side of it, where a decision
from sums against a guess of the rows' maxima would not be safe.  Draft tokens that are the rows' largest logits, those that are not,
and draft rows whose token is far below (its sum against the guess leaves float32's range)."""
import numpy as np
import pytest

from tests.test_gpu_sampling import dev, pool  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 30])           # all positions in one stage, and one by one
@pytest.mark.parametrize("V", [777, 4096, 9001, 50256])       # single loads, and vectors; clusters of one, two, four and eight CTAs
@pytest.mark.parametrize("tokens", ["largest", "drawn", "far"])
def test_decisions_next_to_the_boundary(pool, oracle, n, V, tokens):  # noqa: F811
    rng = np.random.default_rng(V + n + len(tokens))
    k = 4
    dl = (2.5 * rng.standard_normal((n, k, V))).astype(np.float32)
    tl = np.empty((n, k + 1, V), np.float32)
    tl[:, :k] = dl + 0.8 * rng.standard_normal((n, k, V)).astype(np.float32)
    tl[:, k] = 2.5 * rng.standard_normal((n, V)).astype(np.float32)
    if tokens == "largest":
        toks = dl.argmax(axis=2).astype(np.int32)
    else:
        toks = rng.integers(0, V, (n, k)).astype(np.int32)
    if tokens == "far":
        i, j = np.ogrid[:n, :k]
        dl[i, j, toks] = -120.0
        tl[i, j, toks] = -121.0
    cfg = oracle.sampler_cfg()
    probe = np.zeros((n, k + 1), np.float32)     # draws of zero accept everything: all acceptance probabilities
    probe[:, k] = 0.5
    want, draws = [], probe.copy()
    for b in range(n):
        ap = np.asarray(oracle.spec_accept(cfg, toks[b], dl[b], tl[b], probe[b])[3], np.float64)
        stop = rng.integers(0, k + 1)            # accepted up to here, rejected at it
        for i in range(k):
            side = 1.004 if i == stop else 0.996
            draws[b, i] = min(ap[i] * side, 0.99999) if len(ap) > i else 0.0
        want.append(oracle.spec_accept(cfg, toks[b], dl[b], tl[b], draws[b])[0])
    n_acc, _ = pool.spec_accept(n, k, V, toks, dl, tl, draws)
    assert n_acc.tolist() == want
    assert len(set(want)) > 1 or tokens == "far"
