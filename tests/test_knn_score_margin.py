"""CPU checks of the score bounds that the two-scan kNN search rests on
(score_margin, k_bound_kth and k_score_cap in single-clustering_b200/csrc/sc_knn.cu).

The tensor-core score of query x and point y is A(x) . B(y) with 16-bit operands
A = [-2 x^, c1, c2], B = [y^, hi, lo] (k_knn_prep): f16 under a common power of two
where the points' range allows it, BF16 otherwise. The search assumes that it lies
within a Y + b Y^2 of |y|^2 - 2 x.y for |y| <= Y, with a from the measured rounding
errors and b = 2^-13. From that follow a bound on each query's (k+1)-th squared
distance, from 8-column score minima, and a score below which all that can reach
the list must lie. Here the operands are rounded in numpy as the kernel rounds them;
products and sums are in FP64, so half of b stays for the FP32 accumulation: 64
additions, each within 2^-23 of a partial sum of at most 3 Y^2, are 2^-15.4 Y^2."""
import numpy as np
import pytest

import mlp_oracle as mo

B = 2.0 ** -13
KEEP = 16        # minima kept of either half (BOUND_KEEP)
UP = np.float32(1 + 2.0 ** -16)


def f16_exp(X):
    big = np.abs(X).max()
    rows = np.abs(X).max(1)
    rows = rows[rows > 0]
    if not (2.0 ** -40 < big < 2.0 ** 40) or len(rows) == 0 or not rows.min() * 2.0 ** 12 >= big:
        return None
    return 6 - int(np.floor(np.log2(big)))


def operands(X):
    """(x^ in the points' units, B's norm terms' sum, |x|, |x - x^|, rho), as the kernel rounds them."""
    X = X.astype(np.float32)
    e = f16_exp(X)
    nrm = np.zeros(len(X), np.float32)
    for c in X.T:
        nrm = (nrm + c * c).astype(np.float32)
    if e is not None:
        s = np.float32(2.0 ** e)
        back = (X * s).astype(np.float16).astype(np.float32) * np.float32(2.0 ** -e)
        v = (nrm * s * s * np.float32(1 / 32)).astype(np.float32)
        hi = v.astype(np.float16)
        lo = ((v - hi.astype(np.float32)) * np.float32(1024)).astype(np.float16)
        norm_terms = (32.0 * hi.astype(np.float64) + 2.0 ** -5 * lo.astype(np.float64)) * 2.0 ** (-2 * e)
    else:
        back = mo.bf16_round(X).astype(np.float32)
        hi = mo.bf16_round(nrm).astype(np.float32)
        lo = mo.bf16_round((nrm - hi).astype(np.float32))
        norm_terms = hi.astype(np.float64) + lo.astype(np.float64)
    res = np.zeros(len(X), np.float32)
    for c in (X - back).astype(np.float32).T:
        res = (res + c * c).astype(np.float32)
    nx, rx = np.sqrt(nrm) * UP, np.sqrt(res) * UP
    with np.errstate(divide="ignore", invalid="ignore"):
        rho = np.where(nrm > 0, np.sqrt(res) / np.sqrt(nrm) * (UP * UP), np.float32(0)).max()
    return back.astype(np.float64), norm_terms, nx.astype(np.float64), rx.astype(np.float64), float(rho)


def scores(X):
    back, norm_terms, *_ = operands(X)
    return norm_terms[None, :] - 2.0 * back @ back.T


def margin_a(nx, rx, rho):
    return 2.0 * (rx + (nx + rx) * rho) * (1 + 2.0 ** -20)


def kth_bound(X, k):
    """k_bound_kth from the 8-column minima of the two halves of every 128 columns."""
    S = scores(X)
    n = len(X)
    _, _, nx, rx, rho = operands(X)
    cols = np.arange(n)
    out = np.empty(n)
    for i in range(n):
        lists = []
        for half in (0, 1):
            of = cols[(cols // 64) % 2 == half]
            groups = of // 8
            minima = [S[i, of[groups == g]].min() for g in np.unique(groups)]
            lists += sorted(minima)[:KEEP]
        lists.sort()
        if len(lists) < k + 1:
            out[i] = np.inf
            continue
        a = margin_a(nx[i], rx[i], rho)
        p = a + 2 * B * nx[i]
        q = lists[k] + nx[i] ** 2 + a * nx[i] + B * nx[i] ** 2
        disc = p * p + 4 * (1 - B) * q
        d = (p + np.sqrt(max(disc, 0.0))) / (2 * (1 - B))
        out[i] = d * d * (1 + 2.0 ** -14)
    return out


def score_cap(X, kb):
    _, _, nx, rx, rho = operands(X)
    a = margin_a(nx, rx, rho)
    Y = nx + np.sqrt(kb)
    low = nx * (1 - 2.0 ** -15)
    with np.errstate(invalid="ignore"):
        cap = kb - low ** 2 + a * Y + B * Y * Y
    return np.where(np.isnan(cap), np.inf, cap)  # no bound: every score is below it


def points(kind, n, d, rng):
    X = rng.normal(size=(n, d))
    if kind == "mixture":
        X = rng.normal(size=(6, d))[rng.integers(0, 6, n)] * 2 + X * rng.uniform(0.7, 1.5)
    elif kind == "small_rows":
        X[: n // 2] *= 2.0 ** -9
        X[n // 2: n // 2 + 3] = 0.0
    elif kind == "wide":
        X[0] *= 1e6
    elif kind == "one_sign":
        X = np.abs(X)
    elif kind == "midpoints":  # every coordinate just below a midpoint of f16's, then of BF16's, spacing
        X = (1 + 2.0 ** -11 * (1 - 2.0 ** -9)) * 2.0 ** rng.integers(-3, 3, (n, d))
        X[: n // 2] = (1 + 2.0 ** -8 * (1 - 2.0 ** -9)) * 2.0 ** rng.integers(-3, 3, (n // 2, d))
    elif kind == "wide_midpoints":
        X = (1 + 2.0 ** -8 * (1 - 2.0 ** -9)) * 2.0 ** rng.integers(-3, 3, (n, d))
        X[0] *= 2.0 ** 14
    elif kind == "integers":
        X = np.round(3 * X)
        X[:20] = 0.0
    return X


KINDS = ["mixture", "small_rows", "wide", "one_sign", "midpoints", "wide_midpoints", "integers"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("scale", [1.0, 1e-7, 1e9, 1e-13, 1e12])
def test_scores_lie_within_the_margin(kind, scale):
    rng = np.random.Generator(np.random.PCG64(len(kind)))
    worst = 0.0
    for d in (1, 3, 30, 31, 50, 62):
        X = (points(kind, 150, d, rng) * scale).astype(np.float32)
        _, _, nx, rx, rho = operands(X)
        X64 = X.astype(np.float64)
        true = (X64 ** 2).sum(1)[None, :] - 2.0 * X64 @ X64.T
        Y = np.maximum(np.sqrt((X64 ** 2).sum(1))[None, :], np.sqrt((X64 ** 2).sum(1))[:, None])
        room = margin_a(nx, rx, rho)[:, None] * Y + B / 2 * Y * Y
        err = np.abs(scores(X) - true)
        assert np.all(err <= room), (kind, scale, d)
        worst = max(worst, (err[room > 0] / room[room > 0]).max())
    # the worst case of the measured roundings comes close: the margin is tight
    assert kind == "integers" and worst == 0.0 or worst > 0.9 or scale != 1.0


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("scale", [1.0, 1e-7, 1e9, 1e-13, 1e12])
@pytest.mark.parametrize("n,d,k", [(40, 3, 5), (300, 30, 15), (300, 62, 23)])
def test_bounds_hold_what_can_reach_the_list(kind, scale, n, d, k):
    rng = np.random.Generator(np.random.PCG64(n + d + k))
    X = (points(kind, n, d, rng) * scale).astype(np.float32)
    X64 = X.astype(np.float64)
    d2 = ((X64[:, None, :] - X64[None, :, :]) ** 2).sum(2)
    kth = np.sort(d2, axis=1)[:, k]
    kb = kth_bound(X, k)
    assert np.all(kb >= kth)
    # what lies within the bound, and a rounding further (the FP32 distances), scores at most the cap
    reach = d2 <= kth[:, None] * (1 + 2.0 ** -16)
    cap = score_cap(X, kb)
    assert np.all(np.where(reach, scores(X), -np.inf) <= cap[:, None])
