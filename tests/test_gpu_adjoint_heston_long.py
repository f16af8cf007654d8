"""Heston sensitivities on long grids: k_adjoint_heston serves the FP32 grids of
which an SM holds two blocks (1,536 steps) and every FP64 grid the generic
kernel takes up to its shared memory, the generic kernel the others, with the
same outputs on both sides of the line."""
import pytest

import kontracts_gb300 as kx

pytestmark = pytest.mark.gpu

CALL = kx.european_call("X", 100.0, 1.0)
HESTON = kx.heston(100.0, 0.04, 1.5, 0.05, 0.6, -0.7, 0.03, asset="X", scheme="full_truncation")


@pytest.mark.parametrize("prec,steps,kernel", [
    ("fp32", 1536, "k_adjoint_heston"), ("fp32", 1537, "k_adjoint"), ("fp32", 2000, "k_adjoint"),
    ("fp64", 1024, "k_adjoint_heston"), ("fp64", 1624, "k_adjoint_heston"), ("fp64", 1625, "k_adjoint")])
def test_the_kernel_and_its_outputs(monkeypatch, prec, steps, kernel):
    a = CALL.adjoint(HESTON, n_paths=130, seed=3, steps_per_year=steps, precision=prec)
    assert kx.last_launch_stats()["kernel"] == kernel
    monkeypatch.setenv("KX_ADJOINT_KERNEL", "general")
    b = CALL.adjoint(HESTON, n_paths=130, seed=3, steps_per_year=steps, precision=prec)
    assert kx.last_launch_stats()["kernel"] == "k_adjoint"
    assert a.as_dict() == b.as_dict()
