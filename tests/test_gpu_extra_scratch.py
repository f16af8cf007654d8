"""Memory a call can do without (the normals several FP64 walks share, what the
resident American kernels keep beside the stored spots): where there is none
(here: where KX_EXTRA_SCRATCH allows less than the call asks for) the call runs
on the kernels that need none and returns the same bits, and memory taken by
earlier calls is given back."""
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

GBM = [kx.GBM(s0=100.0, sigma=v, r=0.04, asset="X") for v in (0.2, 0.3, 0.4)]
HESTON = [kx.heston(100.0, v, 1.5, 0.04, 0.5, -0.7, 0.03, asset="X") for v in (0.03, 0.04, 0.05)]


@pytest.mark.parametrize("models", [GBM, HESTON], ids=["gbm", "heston"])
def test_walks_draw_their_own_normals(monkeypatch, models):
    cs = [kx.european_call("X", 95.0, 1.0), kx.european_put("X", 100.0, 1.0), kx.european_call("X", 105.0, 1.0)]

    def price():
        r = kx.price_portfolio(cs, models, [100_000] * 3, 7, steps_per_year=63, precision="fp64")
        return [(x.price, x.std_error) for x in r], kx.last_launch_stats()

    a, with_table = price()
    free = torch.cuda.mem_get_info()[0]
    monkeypatch.setenv("KX_EXTRA_SCRATCH", "0")
    b, without = price()
    assert with_table["kernel"] == without["kernel"] == "k_sync"
    assert with_table["kernel_launches"] == without["kernel_launches"] + 1
    assert a == b
    if models is HESTON:  # 101 MB of normals (a GBM European walks one step)
        assert torch.cuda.mem_get_info()[0] - free >= 50_000_000
    monkeypatch.delenv("KX_EXTRA_SCRATCH")
    assert price()[0] == a


@pytest.mark.parametrize("prec,basis", [("fp32", "monomial"), ("fp32", "laguerre"), ("fp64", "monomial"), ("fp64", "laguerre")])
def test_american_without_resident_tiles(monkeypatch, prec, basis):
    put = kx.scale((kx.const_(40.0) - kx.S("X")).clip(0.0), kx.one())
    m = kx.GBM(s0=39.0, sigma=0.3, r=0.06, asset="X")
    dates = [0.1 * i for i in range(1, 11)]

    def price():
        r = put.price_american(m, dates, n_paths=30_001, n_basis=4, basis=basis, precision=prec)
        return (r.price, r.std_error), kx.last_launch_stats()["kernel"]

    a, kernel = price()
    assert kernel == ("k_lsm_tiles64" if prec == "fp64" else "k_lsm_tiles")
    monkeypatch.setenv("KX_EXTRA_SCRATCH", "0")
    b, kernel = price()
    assert kernel == "k_lsm_backward" and a == b
    monkeypatch.delenv("KX_EXTRA_SCRATCH")
    assert price()[0] == a
