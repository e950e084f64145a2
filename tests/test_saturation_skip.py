"""CPU: the rule by which the weighted sweep leaves out the scales that saturate a block, in the kernel's own fp32 operations,
against the plain sweep over every candidate (csrc/quant.cu: sweep_weighted)."""
import numpy as np
import pytest

F = np.float32
E4M3 = np.array([(r & 7) * 2.0 ** -9 if r < 8 else (1 + (r & 7) / 8) * 2.0 ** ((r >> 3) - 7) for r in range(127)], dtype=F)
GRID = np.array([0, .5, 1, 1.5, 2, 3, 4, 6], dtype=F)
EDGES = np.array([.25, .75, 1.25, 1.75, 2.5, 3.5, 5.0], dtype=F)
TIES_UP = np.array([False, True, False, True, False, True, False])   # a tie goes to the even code


def _e2m1(y):
    code = np.zeros(y.shape, dtype=np.int64)
    for edge, up in zip(EDGES, TIES_UP):
        code += (y >= edge) if up else (y > edge)
    return GRID[code]


def _errors(v, w, raw):
    """Weighted squared error of every block at its scale `raw`: the fixed pairwise tree, each operation rounded to fp32."""
    s = E4M3[raw]
    y = np.abs(v) * (F(1) / s)[:, None]
    d = _e2m1(y) - y
    # one rounding of d1^2 * w1 + d0^2 * w0: both products are exact in fp64, as is their sum's rounding to fp32 but for double
    # rounding, which the same expression in the plain sweep shares
    lo = (d[:, 0::2] * d[:, 0::2]) * w[:, 0::2]
    pe = ((d[:, 1::2] * d[:, 1::2]).astype(np.float64) * w[:, 1::2] + lo).astype(F)
    a = pe[:, 0::2] + pe[:, 1::2]
    b = a[:, 0::2] + a[:, 1::2]
    return (b[:, 0] + b[:, 1]) * (s * s)


def _base(v):
    t = np.abs(v).max(1) * np.array([0x3E2AAAAB], dtype=np.uint32).view(F)[0]
    return np.maximum(np.searchsorted(E4M3, t, side="right") - 1, 0)


def _plain(v, w, base, lower, upper):
    best = np.full(len(v), np.inf, dtype=F)
    raw = np.zeros(len(v), dtype=np.int64)
    for off in range(lower, upper + 1):
        cand = np.clip(base + off, 1, 126)
        err = _errors(v, w, cand)
        win = err < best
        best, raw = np.where(win, err, best), np.where(win, cand, raw)
    return raw


def _skipping(v, w, base, lower, upper, exact_weight):
    """One lane's view of the kernel's loop, from the largest scale down; every lane leaves where its own bound allows it (a warp
    leaves only where all of its lanes may: fewer skips, the same rule)."""
    amax = np.abs(v).max(1)
    wmin = w.min(1)
    wb = np.where(wmin >= 0, w[np.arange(len(v)), np.abs(v).argmax(1)], wmin) if exact_weight else wmin
    best = np.full(len(v), np.finfo(F).max, dtype=F)
    raw = np.zeros(len(v), dtype=np.int64)
    alive = np.ones(len(v), dtype=bool)
    skipped = 0
    i = upper - lower
    while i >= 0:
        pair = [i, i - 1] if i > 0 else [i]
        if lower + i < -2 and i < upper - lower:
            s = E4M3[np.clip(base + lower + i, 1, 126)]
            y = amax * (F(1) / s)
            d = F(6) - y
            bound = ((d * d) * wb) * (s * s)
            leave = (base + lower + i < 1) | ((wb >= 0) & (y >= 6) & (y <= 1024) & (best >= F(1e-30)) & (bound > best))
            alive &= ~leave
        for j in pair:
            cand = np.clip(base + lower + j, 1, 126)
            err = _errors(v, w, cand)
            win = alive & (err <= best)
            best, raw = np.where(win, err, best), np.where(win, cand, raw)
        skipped += int((~alive).sum()) * len(pair)
        i -= 2
    return raw, skipped / len(v)


def _blocks(kind, rng, n):
    if kind == "gauss":
        return rng.standard_normal((n, 16)) * 300
    if kind == "laplace":
        return rng.laplace(size=(n, 16)) * 100
    if kind == "equal":
        return np.repeat(rng.uniform(1e-4, 3000, (n, 1)), 16, 1)
    if kind == "single":
        return np.eye(16)[rng.integers(0, 16, n)] * rng.uniform(1e-3, 1e4, (n, 1))
    if kind == "grid":
        return rng.choice([0, .5, 1, 1.5, 2, 3, 4, 6], (n, 16)) * E4M3[rng.integers(1, 127, (n, 1))]
    if kind == "tiny":
        return rng.standard_normal((n, 16)) * 10.0 ** rng.uniform(-44, -2, (n, 1))
    if kind == "huge":
        return rng.standard_normal((n, 16)) * 10.0 ** rng.uniform(3, 37, (n, 1))
    return np.zeros((n, 16))


@pytest.mark.parametrize("window", [(-8, 7), (-3, 7), (-11, 4), (-20, -1), (-20, -5), (-9, -9), (0, 6)])
@pytest.mark.parametrize("kind", ["gauss", "laplace", "equal", "single", "grid", "tiny", "huge", "zero"])
def test_skipping_never_changes_the_chosen_scale(kind, window):
    rng = np.random.default_rng(5)
    n = 600
    v = _blocks(kind, rng, n).astype(F)
    base = _base(v)
    weights = {"even": 1 + 0.05 * rng.standard_normal((n, 16)), "spread": np.exp(2 * rng.standard_normal((n, 16))),
               "zeros": np.where(rng.random((n, 16)) < .5, 0, 1), "small": 10.0 ** rng.uniform(-44, -20, (n, 16)),
               "large": 10.0 ** rng.uniform(20, 38, (n, 16)), "negative": rng.standard_normal((n, 16)),
               "one_negative": np.where(np.arange(16) == 3, -1e-6, 1.0) * np.ones((n, 1))}
    with np.errstate(all="ignore"):
        for name, w in weights.items():
            w = w.astype(F)
            want = _plain(v, w, base, *window)
            for exact_weight in (False, True):
                got, _ = _skipping(v, w, base, *window, exact_weight)
                assert np.array_equal(got, want), (kind, window, name, exact_weight)


def test_most_saturating_scales_are_left_out_with_even_weights():
    rng = np.random.default_rng(6)
    v = _blocks("laplace", rng, 4096).astype(F)
    w = (1 + 0.03 * rng.standard_normal(v.shape)).astype(F)
    assert _skipping(v, w, _base(v), -8, 7, False)[1] > 5.9   # of 16: the pairs -8/-7, -6/-5 and -4/-3
