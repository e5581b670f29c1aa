"""The inverse-CDF search where its levels round differently: the sums of CTAs, warps, lanes and elements are float32 sums of the same
probabilities in different orders, so a draw can lie between two of them.  Whatever level says that the draw is crossed, the token
returned is a neighbour of that point that carries probability, never one with none.

The rows hold one finite logit per warp (or lane), everything else is -inf, so that each sum can be repeated on the host in float32."""
import numpy as np
import pytest

from tests.test_gpu_sampling import dev, pool  # noqa: F401

pytestmark = pytest.mark.gpu

F = np.float32
WARPS, CTAS = 16, 8


def fastexp(x):
    """The reference's fastexp32 (float32 multiply, add, truncation to the bits)."""
    x = np.asarray(x, F)
    t = (F(12102203.0) * np.maximum(x, F(-87.0)) + F(1064948224.0)).astype(F)
    return np.where(x < F(-87.0), F(0.0), t.astype(np.int64).astype(np.uint32).view(F))


def segments(V):
    """First element of every warp's segment, [CTAS][WARPS + 1]."""
    up = lambda a: (a + 127) & ~127   # noqa: E731
    per = up(-(-V // CTAS))
    edges = []
    for q in range(CTAS):
        lo, hi = min(V, q * per), min(V, (q + 1) * per)
        wper = up(-(-(hi - lo) // WARPS))
        edges.append([min(hi, lo + w * wper) for w in range(WARPS + 1)])
    return edges


def in_turn(values):
    a = F(0.0)
    for v in values:
        a = F(a + v)
    return a


def rows_between_cta_and_warps(V, n, seed, masses):
    """Rows [n, V] and draws at which a CTA's scaled sum crosses and its warps' scaled sums do not; the expected tokens.  masses(e):
    what the search sums, of the row's exponentials per warp (flat), as a flat array, and the factor that it applies."""
    rng = np.random.default_rng(seed)
    edges = segments(V)
    full = [(q, w) for q in range(CTAS) for w in range(WARPS) if edges[q][w] < edges[q][w + 1]]
    rows, draws, want = np.full((n, V), -np.inf, F), np.zeros(n, F), np.zeros(n, np.int32)
    for b in range(n):
        while True:
            logit = (-3.0 * rng.random(len(full))).astype(F)
            at = np.array([rng.integers(edges[q][w], edges[q][w + 1]) for q, w in full])
            seg, factor = masses(fastexp(logit - logit.max()), full)
            of = lambda q: [s for s, (c, _) in zip(seg, full) if c == q]   # noqa: E731,B023
            run, hit = F(0.0), None
            for q in range(CTAS):
                base = run
                run = F(run + F(in_turn(of(q)) * factor))
                acc = base
                for s in of(q):
                    acc = F(acc + F(s * factor))
                if 0 < q < CTAS - 1 and acc < run and len(of(q)) < WARPS:
                    hit = (acc, max(a for a, (c, _) in zip(at, full) if c == q))
            if hit:
                break
        rows[b, at] = logit
        draws[b], want[b] = hit
    return rows, draws, want


def cta_order_sum(values, full):
    return in_turn([in_turn([v for v, (c, _) in zip(values, full) if c == q]) for q in range(CTAS)])


@pytest.mark.parametrize("V", [50257, 50256])     # single loads, and vectors; 13 of a CTA's 16 warps have elements
def test_sampled_token_between_the_sums_of_a_cta_and_its_warps(pool, V):  # noqa: F811
    from relux_b200 import lib as L

    def masses(e, full):
        return e, F(F(1.0) / cta_order_sum(e, full))
    rows, draws, want = rows_between_cta_and_warps(V, 16, V, masses)
    pool.tune(L.TUNE_SEL_CLUSTER, CTAS)
    got = pool.sample(rows, draws)
    pool.tune(L.TUNE_SEL_CLUSTER, -1)
    assert np.isfinite(rows[np.arange(len(got)), got]).all(), "a token without probability: %s" % got
    assert got.tolist() == want.tolist()


@pytest.mark.parametrize("V", [50257, 50256])
def test_resampled_token_between_the_sums_of_a_cta_and_its_warps(pool, V):  # noqa: F811
    from relux_b200 import lib as L

    def masses(e, full):      # the draft puts everything on one token that the target rules out: what is left is the target
        t = (e * F(F(1.0) / cta_order_sum(e, full))).astype(F)
        return t, F(F(1.0) / cta_order_sum(t, full))
    rows, r, want = rows_between_cta_and_warps(V, 16, V + 1, masses)
    n = len(rows)
    toks = np.array([int(np.flatnonzero(np.isneginf(x))[7]) for x in rows], np.int32)
    draft = np.full((n, 1, V), -np.inf, F)
    draft[np.arange(n), 0, toks] = 1.0
    target = np.stack([rows, rows], axis=1)
    draws = np.stack([np.full(n, 0.5, F), r], axis=1)
    pool.tune(L.TUNE_SEL_CLUSTER, CTAS)
    n_acc, got = pool.spec_accept(n, 1, V, toks[:, None], draft, target, draws)
    pool.tune(L.TUNE_SEL_CLUSTER, -1)
    assert n_acc.tolist() == [0] * n
    assert np.isfinite(rows[np.arange(n), got]).all(), "a token without probability: %s" % got
    assert got.tolist() == want.tolist()


def lanes_that_cross_without_probability(n, seed, V, per_lane):
    """Rows of V <= 128 (one warp) whose scan over the lanes rounds up at a lane without probability, and the draws below that."""
    rng = np.random.default_rng(seed)
    rows, draws, want = np.full((n, V), -np.inf, F), np.zeros(n, F), np.zeros(n, np.int32)
    lanes = V // 4
    for b in range(n):
        while True:
            has = rng.random(lanes) < 0.6
            at = 4 * np.flatnonzero(has) + rng.integers(0, 4, has.sum())
            logit = (-3.0 * rng.random(len(at))).astype(F)
            e = fastexp(logit - logit.max())
            part = np.zeros(32, F)      # the warp's sum, a butterfly over what its lanes have read
            if per_lane == 4:
                part[np.flatnonzero(has)] = e
            else:
                for j in range(0, V, 32):
                    inside = (at >= j) & (at < j + 32)
                    part[at[inside] - j] = (part[at[inside] - j] + e[inside]).astype(F)
            for o in (16, 8, 4, 2, 1):
                part = (part + part[np.arange(32) ^ o]).astype(F)
            factor = F(F(1.0) / part[0])
            x = np.zeros(32, F)
            x[np.flatnonzero(has)] = (e * factor).astype(F)
            for o in (1, 2, 4, 8, 16):
                x = np.concatenate([x[:o], (x[o:] + x[:-o]).astype(F)])
            top = np.maximum.accumulate(x)
            odd = [j for j in range(1, lanes - 1) if not has[j] and x[j] > top[j - 1] > 0 and top[-1] > x[j]]
            if odd:
                break
        rows[b, at] = logit
        draws[b], want[b] = top[odd[0] - 1], at[at > 4 * odd[0]].min()   # the next one adds what takes the sum past the draw
    return rows, draws, want


@pytest.mark.parametrize("V,per_lane", [(128, 4), (127, 1)])     # vectors, and single loads
def test_sampled_token_where_a_lane_without_probability_crosses(pool, V, per_lane):  # noqa: F811
    rows, draws, want = lanes_that_cross_without_probability(16, V, V - V % 4, per_lane)
    rows = np.concatenate([rows, np.full((16, V % 4), -np.inf, F)], axis=1)
    got = pool.sample(rows, draws)
    assert np.isfinite(rows[np.arange(len(got)), got]).all(), "a token without probability: %s" % got
    assert got.tolist() == want.tolist()
