"""A book's group of several launches reports the shape of its largest one."""
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu


def test_group_of_three_launches():
    m = kx.GBM(s0=100.0, sigma=0.3, r=0.03, asset="X")
    call = kx.european_call("X", 100.0, 1.0)                      # k_sync
    ko = kx.up_and_out_call("X", 100.0, 130.0, 1.0)               # k_knock
    late = kx.scale((kx.S("X") - 100.0).clip(0.0), kx.one()).when(kx.at(1.0)).until(kx.S("X") >= 130.0).when(kx.at(0.5))  # k_lean
    strip = kx.european_call("X", 100.0, 0.3) + kx.european_put("X", 105.0, 1.0)  # k_sync, several steps

    def items(cs, ns):
        book = kx.Book(cs, [m] * len(cs), ns, list(range(len(cs))), steps_per_year=256, tune=False)
        info = book.info()
        book.close()
        assert info["n_groups"] == 1 and info["groups"][0]["contracts"] == len(cs)
        return info["groups"][0]["item_paths"]

    # launch order k_sync, k_knock, k_lean; the most path steps first (6.0M), in the middle and last (768M)
    assert items([strip, ko, late], [3_000_000, 1000, 10_000]) == items([strip], [3_000_000])
    assert items([call, ko, late], [1000, 3_000_000, 40_000]) == items([ko], [3_000_000])
    assert items([call, ko, late], [40_000, 1000, 3_000_000]) == items([late], [3_000_000])
