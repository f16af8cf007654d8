"""k_adjoint_heston (threads in step, segments in registers) gives the generic
adjoint kernel's outputs bit for bit: path counts around a block, grids around
a Philox block (2 steps) and a segment (4 or 8 steps), several flows and a flow at
t = 0, unequal steps, both variance schemes, a portfolio of uneven contracts."""
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu

CONTRACTS = {
    "call": lambda: kx.european_call("X", 100.0, 1.0),
    "strip": lambda: kx.european_call("X", 100.0, 0.31) + kx.european_put("X", 105.0, 0.61) + kx.forward("X", 95.0, 1.0),
    "same_day": lambda: kx.straddle("X", 100.0, 0.5) + kx.scale(kx.S("X"), kx.one()),
    "bond": lambda: kx.zero_coupon_bond("USD", 0.7),
}


def _model(scheme):
    return kx.heston(100.0, 0.04, 1.5, 0.05, 0.6, -0.7, 0.03, asset="X", scheme=scheme)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("scheme", ["reference", "full_truncation"])
@pytest.mark.parametrize("name", sorted(CONTRACTS))
def test_equals_the_generic_kernel(monkeypatch, name, scheme, prec):
    c, m = CONTRACTS[name](), _model(scheme)
    for n, spy in ((1, 1), (127, 2), (129, 7), (64, 8), (300, 9), (1000, 63), (200, 252), (40, 600)):
        a = c.adjoint(m, n_paths=n, seed=3, steps_per_year=spy, precision=prec)
        monkeypatch.setenv("KX_ADJOINT_KERNEL", "general")
        b = c.adjoint(m, n_paths=n, seed=3, steps_per_year=spy, precision=prec)
        monkeypatch.delenv("KX_ADJOINT_KERNEL")
        assert a.as_dict() == b.as_dict(), (n, spy)


def test_portfolio_equals_the_generic_kernel(monkeypatch):
    cs = [CONTRACTS[k]() for k in sorted(CONTRACTS)]
    ms = [_model("reference"), _model("full_truncation"), _model("reference"), _model("full_truncation")]
    args = (cs, ms, [130, 1, 777, 256], [1, 2, 3, 4])
    _, a = kx.price_portfolio(*args, steps_per_year=100, greeks=True)
    monkeypatch.setenv("KX_ADJOINT_KERNEL", "general")
    _, b = kx.price_portfolio(*args, steps_per_year=100, greeks=True)
    assert [x.as_dict() for x in a] == [x.as_dict() for x in b]
