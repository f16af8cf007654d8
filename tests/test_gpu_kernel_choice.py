"""Which kernel serves a call: the contracts whose values other tests compare
between kernels run on the kernel those tests are about."""
import pytest
import test_gpu_adjoint_heston as heston
import test_gpu_knock as knock
import test_gpu_multi_knock as multi
import test_gpu_one_draw as one_draw
import test_gpu_sync as sync
import test_gpu_tangent_walk as tangent

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu


def _kernel():
    return kx.last_launch_stats()["kernel"]


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_static_schedules(monkeypatch, prec):
    for name, c in sorted(sync.CONTRACTS.items()):
        for m in (sync.GBM, sync.HESTON):
            c().price(m, n_paths=33, steps_per_year=63, precision=prec)
            assert _kernel() == "k_sync", name
    for choice, want in (("lean", "k_lean"), ("general", "k_paths")):
        monkeypatch.setenv("KX_PATH_KERNEL", choice)
        sync.CONTRACTS["call"]().price(sync.GBM, n_paths=33, steps_per_year=63, precision=prec)
        assert _kernel() == want


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_knock_outs_and_knock_ins(prec):
    m = kx.GBM(s0=100.0, sigma=0.3, r=0.04, asset="X")
    for name, c in sorted(knock.CONTRACTS.items()):
        for spy in (2, 64, 1024, 1025):
            c().price(m, n_paths=33, steps_per_year=spy, precision=prec)
            assert _kernel() == ("k_knock" if name != "in_early_flow" and spy <= 1024 else "k_lean"), (name, spy)


@pytest.mark.parametrize("window", [(0.0, 1.0, 1.0), (0.26, 0.74, 1.0)])
def test_averages_on_one_draw(window):
    """The sizes of test_gpu_one_draw fill this device with groups of seven walks."""
    c = one_draw._asian(*window)
    for k in (5, 7, 15):
        kx.price_portfolio([c] * k, one_draw._models(k), [one_draw.N] * k, 5, steps_per_year=63)
        assert _kernel() == "k_sync_scen"
    kx.price_portfolio([c] * 4, one_draw._models(4), [one_draw.N] * 4, 5, steps_per_year=63)
    assert _kernel() == "k_sync"


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_normals_drawn_once(prec):
    """FP64 walks of one stream read a table of its normals: one launch more."""
    cs = [sync.CONTRACTS["call"]()] * 3
    ms = [kx.GBM(s0=100.0, sigma=v, r=0.04, asset="X") for v in (0.2, 0.3, 0.4)]
    kx.price_portfolio(cs, ms, [2050] * 3, 7, steps_per_year=63, precision=prec)
    st = kx.last_launch_stats()
    assert st["kernel"] == "k_sync" and st["kernel_launches"] == (3 if prec == "fp64" else 2)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_correlated_factors(prec):
    for name, c in sorted(multi.CONTRACTS.items()):
        for n in (2, 5, 7):
            c(n).price(multi._model(n), n_paths=33, steps_per_year=4, precision=prec)
            assert _kernel() == "k_multi_knock", (name, n)


def test_shared_simulation():
    cs = [kx.european_call("X", k, t) for k in (90.0, 110.0) for t in (0.5, 1.0)]
    for m in (sync.GBM, sync.HESTON):
        for prec in ("fp32", "fp64"):
            kx.price_batch(cs, m, n_paths=300, steps_per_year=63, precision=prec)
            assert _kernel() == "k_flows_walk"


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_heston_adjoint(prec):
    for name, c in sorted(heston.CONTRACTS.items()):
        for spy in (1, 9, 252, 600):
            c().adjoint(heston._model("reference"), n_paths=40, steps_per_year=spy, precision=prec)
            assert _kernel() == "k_adjoint_heston", (name, spy)


def test_gbm_adjoint():
    for name, c in sorted(tangent.CONTRACTS.items()):
        for spy in (4, 64, 1024):
            c().adjoint(tangent.GBM, n_paths=40, steps_per_year=spy)
            assert _kernel() == "k_tangent_walk", (name, spy)
    c().adjoint(tangent.GBM, n_paths=40, steps_per_year=64, precision="fp64")
    assert _kernel() != "k_tangent_walk"


def test_american_options():
    put = kx.scale((kx.const_(40.0) - kx.S("X")).clip(0.0), kx.one())
    m = kx.GBM(s0=36.0, sigma=0.2, r=0.06, asset="X")
    for prec, want in (("fp32", "k_lsm_tiles"), ("fp64", "k_lsm_tiles64")):
        put.price_american(m, [0.25, 0.5, 0.75, 1.0], n_paths=20_000, precision=prec)
        assert _kernel() == want
