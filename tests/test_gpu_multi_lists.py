"""k_multi_knock gives k_multi_lean's values (KX_PATH_KERNEL=lean) bit for bit:
the contracts of its comparison with the general kernel, on grids whose steps
are equal in both precisions."""
import numpy as np
import pytest
import test_gpu_multi_knock as multi

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("name", sorted(multi.CONTRACTS))
def test_equals_the_event_handler(monkeypatch, name, prec):
    for n_a, n, spy in [(2, 1, 1), (3, 31, 2), (4, 33, 4), (5, 257, 8), (6, 600, 32), (7, 1030, 16), (5, 300, 256), (2, 20_000, 8)]:
        c, m = multi.CONTRACTS[name](n_a), multi._model(n_a)
        r, p = c.price(m, n_paths=n, seed=8, steps_per_year=spy, precision=prec, per_path=True)
        assert kx.last_launch_stats()["kernel"] == "k_multi_knock"
        monkeypatch.setenv("KX_PATH_KERNEL", "lean")
        s, q = c.price(m, n_paths=n, seed=8, steps_per_year=spy, precision=prec, per_path=True)
        assert kx.last_launch_stats()["kernel"] == "k_multi_lean"
        monkeypatch.delenv("KX_PATH_KERNEL")
        assert np.array_equal(np.asarray(p), np.asarray(q)) and r.price == s.price, (n_a, n, spy)

