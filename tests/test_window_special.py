"""Fits of BOLD whose correlations are not ordinary numbers: constant nodes (also
in some windows only), NaN and infinite values, variances far outside the usual
range.  The flag that turns such a series' cost into the maximum, and the values
of the pairs and series that are not concerned, are checked against the oracle,
which is plain FP64 (GPU)."""
import numpy as np
import pytest

import bnm_cuda_b200 as B

N, FRAMES, SIZE, STEP = 37, 70, 8, 2  # three node tiles, the last one ragged; windows ending inside and across chunks


def _series(rng):
    z = rng.standard_normal((FRAMES + 4, N))
    return sum(z[k:k + FRAMES] for k in range(5)).astype(np.float32).astype(np.float64)


def _mixed(kind, rng, f64):
    """One series of the given kind and the nodes whose pairs it concerns."""
    x = _series(rng)
    if kind == "constant":
        x[:, 20] = 1.25
    elif kind == "zero":
        x[:, 0] = 0.0
    elif kind == "constant_window":  # zero over the frames of some windows; whole numbers of mean 0, so sums are exact
        x[:, 33] = rng.integers(-9, 10, FRAMES)
        x[20:34, 33] = 0.0
        x[0, 33] -= x[:, 33].sum()
        return x, [33]
    elif kind == "nan":
        x[41, 5] = np.nan
        return x, [5]
    elif kind == "nan_last":
        x[FRAMES - 1, N - 1] = np.nan
        return x, [N - 1]
    elif kind == "inf":
        x[3, 16] = np.inf
        return x, [16]
    elif kind in ("huge", "tiny"):  # finite; products of these variances leave FP32's range, not FP64's
        x *= 2.0 ** ((240 if f64 else 60) * (1 if kind == "huge" else -1))
        return x, []
    return x, [20] if kind == "constant" else [0]


def _pearson(x, i, j):
    z = x - x.mean(0)
    return (z[:, i] * z[:, j]).sum(0) / (np.sqrt((z[:, i] ** 2).sum(0)) * np.sqrt((z[:, j] ** 2).sum(0)))


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [B.PREC_F32, B.PREC_F64])
@pytest.mark.parametrize("kind", ["constant", "zero", "constant_window", "nan", "nan_last", "inf", "huge", "tiny"])
def test_special_values_match_oracle(port, kind, prec):
    rng = np.random.default_rng(5)
    special, nodes = _mixed(kind, rng, prec == B.PREC_F64)
    bold = np.stack([_series(rng), special, _series(rng)])
    cfg = B.Config(nodes=N, max_sims=3, time_steps=1000 * (FRAMES - 1), bold_tr=1000, bold_remove_s=0, window_size=SIZE,
                   window_step=STEP, exc_interhem=False, precision=prec, gram=B.GRAM_F32)
    emp_fc, emp_fcd = rng.uniform(-0.2, 0.8, cfg.sizes()["n_pairs"]), rng.uniform(-0.2, 0.9, 100)
    with B.Plan(cfg, np.zeros((N, N)), emp_fc, emp_fcd) as p:
        r = p.check_fit_bold(bold)
        again = p.check_fit_bold(bold[[0, 2, 0]])  # the flag does not outlive its call
    i, j = np.tril_indices(N, -1)
    sound = ~(np.isin(i, nodes) | np.isin(j, nodes))
    for s in range(3):
        on = sound if s == 1 else np.ones_like(sound)
        # FP64, rounded once to FP32
        np.testing.assert_allclose(r["fc"][s][on], _pearson(bold[s], i[on], j[on]), rtol=2e-7, atol=1e-7)
    ordinary = kind in ("huge", "tiny")
    if not ordinary:
        assert r["cost"][1] == cfg.max_cost
    for s in (0, 1, 2) if ordinary else (0, 2):
        want = port.port_gof(bold[s], STEP, SIZE, emp_fc, np.sort(emp_fcd), False)
        assert r["cost"][s] == pytest.approx(want["cost"], abs=1e-5)  # one KS jump is 1e-2
    np.testing.assert_array_equal(again["cost"], r["cost"][[0, 2, 0]])
