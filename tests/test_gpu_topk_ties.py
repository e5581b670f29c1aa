"""Top-k of long rows whose ties put many lanes of a warp on the list, or the whole row over it: on either side of the number of lanes
that a warp goes through one by one, rows that are read four at a time and one by one, lists narrowed down by the radix walk, and rows of
equal logits or of few finite ones."""
import numpy as np
import pytest

from tests.test_gpu_sampling import dev, pool  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [131072, 131071, 40000])
@pytest.mark.parametrize("kind", ["plateau 60", "plateau 300", "plateau 700", "block 200", "steps", "equal", "few finite"])
def test_ties_of_long_rows(pool, oracle, V, kind):  # noqa: F811
    rng = np.random.default_rng(V + len(kind))
    rows, top_k = 3, 50
    x = (2.5 * rng.standard_normal((rows, V))).astype(np.float32)
    name, _, count = kind.partition(" ")
    if name == "plateau":                       # ties at the top, spread over the row
        for row in x:
            row[rng.permutation(V)[:int(count)]] = 20.0
    elif name == "block":                       # ties side by side: every lane of a few warps
        for i, row in enumerate(x):
            row[1000 * i + 7:1000 * i + 7 + int(count)] = 20.0
    elif name == "steps":
        x = np.round(4 * x) / 4
    elif name == "equal":
        x[:] = 1.25
    else:
        x[:, 40:] = -np.inf
    # Where the list does not hold the ties, a nucleus cut between equal probabilities keeps all of them and sums run in another order:
    # no nucleus there, and every draw lies in the middle of a token's interval.
    top_p = 1.0 if kind in ("plateau 700", "equal") else 0.95
    cfg = oracle.sampler_cfg(temperature=0.8, top_k=top_k, top_p=top_p)
    want, draws = [], []
    for row in x:
        probs = oracle.sampler_sample(cfg, row, 0.5, return_probs=True)[1]
        cum, kept = np.cumsum(probs.astype(np.float64)), np.flatnonzero(probs > 0)
        want.append(int(kept[int(len(kept) * rng.random())]))
        draws.append(cum[want[-1]] - probs[want[-1]] / 2)
    got = pool.sample(x, np.asarray(draws, np.float32), temperature=0.8, top_k=top_k, top_p=top_p)
    # V equal probabilities: float32 sums of up to V terms are off by V * 2^-24 of themselves at most, V times that many tokens
    slack = V * V * 2.0 ** -24 if kind == "equal" else 0
    assert np.abs(got - np.asarray(want)).max() <= slack, (got, want)
