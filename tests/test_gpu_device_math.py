"""The engine's device arithmetic against CUDA's own functions, over whole
ranges of inputs: tests/cuda/device_math.cu is compiled with the engine's
headers and counts the inputs on which the two differ."""
import ctypes as C
import os
import struct
import subprocess

import pytest

from kontracts_gb300 import build as kb

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def _bits(x):
    return struct.unpack("<I", struct.pack("<f", x))[0]


@pytest.fixture(scope="module")
def dev(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("device_math") / "device_math.so")
    subprocess.run([kb._nvcc(), *kb.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC,-ffp-contract=off",
                    "--expt-relaxed-constexpr", "-I", kb.INCLUDE, "-shared", "-o", out,
                    os.path.join(HERE, "cuda", "device_math.cu")], check=True)
    lib = C.CDLL(out)

    def call(name, *args):
        f = getattr(lib, name)
        f.restype = C.c_longlong
        return f(*args)

    return call


def test_regression_weight_keeps_its_last_bits(dev):
    """e^(-x/2) for every FP32 x of [0, 256): nothing is flushed to zero where the weight is subnormal
    (spots of 175 to 208 times the model's)."""
    top = _bits(256.0)
    assert dev("check_basis_weight", C.c_uint32(0), C.c_uint32(top)) == 0


def test_normals_are_those_of_the_library_logarithm(dev):
    """All 2^32 first words of a Box-Muller pair."""
    assert dev("check_normal_pairs") == 0


@pytest.mark.parametrize("sign,limit", [(0, 200.0), (1, 80.0)])
def test_exponential_without_subnormal_results(dev, sign, limit):
    """e^y for every FP32 y of [-80, 200), the infinite results among them."""
    assert dev("check_tame_exp", C.c_uint32(sign), C.c_uint32(0), C.c_uint32(_bits(limit) + 1)) == 0


@pytest.mark.parametrize("kind", ["spread", "tie_76_bits", "tie_77_bits", "beside_a_tie", "carry", "amounts", "factors"])
def test_discounted_amount_is_the_fp64_product(dev, kind):
    """16M pairs of a kind, bit for bit (any NaN for a NaN)."""
    kinds = ["spread", "tie_76_bits", "tie_77_bits", "beside_a_tie", "carry", "amounts", "factors"]
    assert dev("check_discount", C.c_int(kinds.index(kind)), C.c_uint32(1 << 24)) == 0
