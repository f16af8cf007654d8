"""The table of normals that FP64 walks of one stream share holds the draws of
their grid and no more: walks whose last Philox block holds one, two or three
draws, tables that end at and beside the 2 MiB granules of device memory. Every
price equals the contract's own call."""
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu

S = kx.S("X")
ASIAN = kx.scale((kx.average(S) - 100.0).clip(0.0), kx.one()) @ kx.at(1.0)
CALL = kx.european_call("X", 100.0, 1.0)
GBM = [kx.GBM(s0=100.0, sigma=v, r=0.04, asset="X") for v in (0.2, 0.3)]
HESTON = [kx.heston(100.0, v, 1.5, 0.04, 0.5, -0.7, 0.03, asset="X") for v in (0.03, 0.04)]
GRANULE = (2 << 20) // 8  # doubles


@pytest.mark.parametrize("contract,models,spy,draws", [
    (CALL, GBM, 7, 1), (ASIAN, GBM, 1, 1), (ASIAN, GBM, 2, 2), (ASIAN, GBM, 3, 3), (ASIAN, GBM, 4, 4), (ASIAN, GBM, 5, 5),
    (ASIAN, GBM, 9, 9), (ASIAN, GBM, 33, 33), (CALL, HESTON, 1, 2), (CALL, HESTON, 3, 6), (ASIAN, HESTON, 5, 10)])
def test_tables_end_where_the_grid_does(monkeypatch, contract, models, spy, draws):
    monkeypatch.setenv("KX_EXTRA_SCRATCH", "0")  # gives an earlier, larger table back
    kx.price_portfolio([contract] * 2, models, [100] * 2, 5, steps_per_year=spy, precision="fp64")
    monkeypatch.delenv("KX_EXTRA_SCRATCH")
    for n in sorted({1, 31, 100, GRANULE // draws, GRANULE // draws + 1}):
        got = kx.price_portfolio([contract] * 2, models, [n] * 2, 5, steps_per_year=spy, precision="fp64")
        assert kx.last_launch_stats()["kernel_launches"] == 3  # the table, the walks, the statistics
        for m, r in zip(models, got):
            assert r.price == contract.price(m, n_paths=n, seed=5, steps_per_year=spy, precision="fp64").price
