"""The American pricer's backward kernels agree bit for bit in each precision:
blocks that keep a tile or a part of one, every block solving (calls whose
tiles are all resident), and blocks that walk over several tiles with
coordinators (larger calls). The same case is priced alone and in a batch that
a second, large case makes too large for the first kernel; sums, solves and decisions take the same order in
both, so the results are equal, at the edges of a group of paths, of a tile
and of the gather over tiles, for each basis size, basis and payoff form."""
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu

TILE = 8192
PAYOFFS = {
    "put": lambda: kx.scale((kx.const_(40.0) - kx.S("X")).clip(0.0), kx.one()),
    "call": lambda: kx.scale((kx.S("X") - 38.0).clip(0.0), kx.one()),
    "spot": lambda: kx.scale(kx.S("X"), kx.one()),
    "two_terms": lambda: kx.scale((kx.const_(42.0) - kx.S("X")).clip(0.0), kx.one())
    + kx.give(kx.scale((kx.const_(38.0) - kx.S("X")).clip(0.0), kx.one())),
    "cash": lambda: kx.scale(kx.const_(2.0), kx.one()),
}


def _dates(t, n):
    return [t * i / n for i in range(1, n + 1)]


def _check(cases, basis, n_basis, precision="fp32"):
    filler = (PAYOFFS["put"](), kx.GBM(s0=40.0, sigma=0.2, r=0.06, asset="X"), [0.5, 1.0], 400 * TILE, 9)
    batch = kx.price_american_batch(cases + [filler], n_basis=n_basis, basis=basis, precision=precision)
    for (c, m, ds, n, seed), b in zip(cases, batch):
        a = c.price_american(m, ds, n_paths=n, seed=seed, n_basis=n_basis, basis=basis, precision=precision)
        assert (a.price, a.std_error, a.n_paths) == (b.price, b.std_error, b.n_paths), (n, len(ds))


@pytest.mark.parametrize("basis", ["monomial", "laguerre"])
@pytest.mark.parametrize("n_basis", [2, 3, 4, 5, 6])
def test_sizes(basis, n_basis):
    m = kx.GBM(s0=39.0, sigma=0.3, r=0.06, asset="X")
    sizes = (1, 3, 255, 1024, 1025, 2047, 2049, TILE - 1, TILE, TILE + 1, 5 * TILE + 700, 17 * TILE, 129 * TILE + 5)
    _check([(PAYOFFS["put"](), m, _dates(1.0, 7), n, 3 + n) for n in sizes], basis, n_basis)


@pytest.mark.parametrize("name", sorted(PAYOFFS))
@pytest.mark.parametrize("n_dates", [1, 2, 3, 50])
def test_payoffs_and_dates(name, n_dates):
    gbm = kx.GBM(s0=41.0, sigma=0.25, r=0.05, asset="X")
    heston = kx.heston(40.0, 0.05, 2.0, 0.05, 0.4, -0.6, 0.05, asset="X")
    _check([(PAYOFFS[name](), gbm, _dates(1.0, n_dates), 20_001, 5),
            (PAYOFFS[name](), heston, _dates(0.7, n_dates), 9_000, 6)], "monomial", 3)


def test_many_small_cases_in_one_call():
    cases = [(PAYOFFS["put"](), kx.GBM(s0=36.0 + 0.1 * i, sigma=0.2, r=0.06, asset="X"), _dates(1.0, 3 + i % 9),
              700 + 311 * i, i) for i in range(90)]
    got = kx.price_american_batch(cases, n_basis=4, basis="laguerre")
    for (c, m, ds, n, seed), b in list(zip(cases, got))[::7]:
        a = c.price_american(m, ds, n_paths=n, seed=seed, n_basis=4, basis="laguerre")
        assert (a.price, a.std_error) == (b.price, b.std_error), n


@pytest.mark.parametrize("basis", ["monomial", "laguerre"])
@pytest.mark.parametrize("n_basis", [2, 3, 4, 5, 6])
def test_sizes_fp64(basis, n_basis):
    m = kx.GBM(s0=39.0, sigma=0.3, r=0.06, asset="X")
    sizes = (1, 31, 33, 255, 1025, TILE - 1, TILE, TILE + 1, 2 * TILE + 700, 17 * TILE, 38 * TILE)
    _check([(PAYOFFS["put"](), m, _dates(1.0, 5), n, 3 + n) for n in sizes], basis, n_basis, "fp64")


@pytest.mark.parametrize("name", sorted(PAYOFFS))
@pytest.mark.parametrize("n_dates", [1, 2, 3, 25])
def test_payoffs_and_dates_fp64(name, n_dates):
    gbm = kx.GBM(s0=41.0, sigma=0.25, r=0.05, asset="X")
    heston = kx.heston(40.0, 0.05, 2.0, 0.05, 0.4, -0.6, 0.05, asset="X")
    _check([(PAYOFFS[name](), gbm, _dates(1.0, n_dates), 20_001, 5),
            (PAYOFFS[name](), heston, _dates(0.7, n_dates), 9_000, 6)], "laguerre", 3, "fp64")
