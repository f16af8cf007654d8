"""k_multi_knock (correlated factors, knock-outs without an event handler)
against the general kernel on the same paths: 2 to 7 factors, path counts around
a warp, a group of warps and a block's list, grids around a round of 4 steps and
a segment, one to three barrier rows of every comparison, flows at t = 0 and
several at the last date, a path knocked out at t = 0, no barrier at all.
Tolerances as the affine kernel's: 1e-12 (FP64) and 1e-6 (FP32) of
max(|value|, 100); the FP32 runs are too few paths to come within rounding of a
barrier."""
import numpy as np
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu


def _model(n):
    fac = [(f"A{i}", 100.0 - i, 0.03, 0.15 + 0.04 * i) for i in range(n)]
    return kx.CorrelatedGbmN(fac, [[1.0 if i == j else 0.3 for j in range(n)] for i in range(n)], rate=0.02)


def _basket(n):
    b = kx.S("A0")
    for i in range(1, n):
        b = b + kx.S(f"A{i}")
    return b / float(n)


def _call(n, k=98.0):
    return kx.scale((_basket(n) - k).clip(0.0), kx.one()) @ kx.at(1.0)


CONTRACTS = {
    "up_out": lambda n: kx.until(_basket(n) >= 112.0, _call(n)),
    "down_out_strict": lambda n: kx.until(kx.S("A1") < 85.0, _call(n)),
    "double_and_spread": lambda n: kx.until(_basket(n) > 115.0, kx.until(_basket(n) <= 85.0, kx.until(
        kx.S("A0") - kx.S("A1") >= 30.0, _call(n) + kx.scale(kx.S("A1"), kx.one()) @ kx.at(1.0)))),
    "with_a_flow_now": lambda n: kx.one() + kx.until(_basket(n) >= 115.0, _call(n)),
    "knocked_at_zero": lambda n: kx.until(_basket(n) >= 50.0, _call(n)),
    "european": lambda n: _call(n) + kx.give(kx.scale((95.0 - kx.S("A0")).clip(0.0), kx.one()) @ kx.at(1.0)),
}


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("name", sorted(CONTRACTS))
def test_equals_the_general_kernel(monkeypatch, name, prec):
    shapes = [(2, 1, 1), (3, 31, 3), (4, 33, 4), (5, 257, 9), (6, 600, 30), (7, 1030, 13), (5, 300, 252)]
    if prec == "fp64":
        shapes += [(2, 20_000, 10), (7, 5_000, 6)]
    for n_a, n, spy in shapes:
        c, m = CONTRACTS[name](n_a), _model(n_a)
        _, p = c.price(m, n_paths=n, seed=8, steps_per_year=spy, precision=prec, per_path=True)
        assert kx.last_launch_stats()["path_kernel"] == 5
        monkeypatch.setenv("KX_PATH_KERNEL", "general")
        _, q = c.price(m, n_paths=n, seed=8, steps_per_year=spy, precision=prec, per_path=True)
        monkeypatch.delenv("KX_PATH_KERNEL")
        p, q = np.asarray(p), np.asarray(q)
        tol = 1e-12 if prec == "fp64" else 1e-6
        assert np.all(np.abs(p - q) <= tol * np.maximum(np.abs(q), 100.0)), (n_a, n, spy)
