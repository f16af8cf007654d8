"""American options of few dates: small calls stay on k_lsm_backward, at both
sides of the line the kernels agree bit for bit."""
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("basis,n_basis", [("monomial", 2), ("laguerre", 4)])
@pytest.mark.parametrize("prec,n,dates,tiles", [
    ("fp32", 1, 1, False), ("fp32", 1024, 3, False), ("fp32", 1025, 3, True), ("fp32", 1025, 1, True), ("fp32", 33, 4, True),
    ("fp64", 1024, 2, False), ("fp64", 1025, 2, True), ("fp64", 2049, 1, True), ("fp64", 409, 5, False), ("fp64", 33, 6, True)])
def test_the_line(monkeypatch, prec, n, dates, tiles, basis, n_basis):
    put = kx.scale((kx.const_(40.0) - kx.S("X")).clip(0.0), kx.one())
    m = kx.GBM(s0=39.0, sigma=0.3, r=0.06, asset="X")
    ds = [1.0 * i / dates for i in range(1, dates + 1)]
    a = put.price_american(m, ds, n_paths=n, seed=5, n_basis=n_basis, basis=basis, precision=prec)
    kernel = kx.last_launch_stats()["kernel"]
    assert kernel == ("k_lsm_tiles64" if prec == "fp64" else "k_lsm_tiles") if tiles else kernel == "k_lsm_backward"
    monkeypatch.setenv("KX_EXTRA_SCRATCH", "0")
    b = put.price_american(m, ds, n_paths=n, seed=5, n_basis=n_basis, basis=basis, precision=prec)
    assert kx.last_launch_stats()["kernel"] == "k_lsm_backward"
    assert a.price == b.price and a.n_paths == b.n_paths
    assert a.std_error == b.std_error or n == 1  # one path has no standard error (nan)
