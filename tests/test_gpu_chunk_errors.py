"""kx_price_chunks hands out nothing when the paths report an error."""
import ctypes as C

import pytest

import kontracts_gb300 as kx
from kontracts_gb300 import _abi

pytestmark = pytest.mark.gpu


def test_an_error_of_the_paths_leaves_the_output_alone():
    # an average read before its window closes: known on the device alone when the read waits for a price
    S = kx.S("X")
    c = kx.when(S >= 50.0, kx.scale(kx.average_over(S, 0.0, 0.9), kx.one())) + kx.zero_coupon_bond("USD", 1.0)
    m = kx.GBM(s0=100.0, sigma=0.2, r=0.02, asset="X")
    h = c._handle()
    cm, cfg = m._c(), kx._cfg(1000, 7, 50, m.rate, "fp32", False)
    out = (_abi.KxChunkStats * 4)()
    for o in out:
        o.n, o.mean, o.m2 = -1.0, -2.0, -3.0
    n_out = C.c_size_t(99)
    st = kx._lib().kx_price_chunks(h.h, C.byref(cm), C.byref(cfg), 0, out, 4, C.byref(n_out))
    assert st == _abi.KX_UNSUPPORTED
    assert n_out.value == 99 and all((o.n, o.mean, o.m2) == (-1.0, -2.0, -3.0) for o in out)
