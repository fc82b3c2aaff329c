"""The flux kernel above the sizes that give a thread one face (choose_march marches on once a face a thread is more
than the GPU's threads, at most 132,608 on 148 SMs): marches of several faces along y and z, cut into chunks of unequal
length, x CTAs of two to four groups of cells, ragged in every direction. The plain form steps to the oracle's
bits, the FP32-flux form stays within 1e-5 of it (relative L1 of the density and the number density), as at the
small sizes (test_gpu_faces.py)."""
import numpy as np
import pytest

from ice_b200 import abi
from test_gpu_faces import _case, _steps, gpu  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("closure,dims,join", [("IG", (88, 87, 90), None), ("AG", (64, 61, 67), 2),
                                               ("MK", (300, 9, 257), 0), ("MK", (797, 701, 1), None)],
                         ids=lambda x: x if isinstance(x, str) else "x".join(map(str, x)) if isinstance(x, tuple) else f"join{x}")
def test_long_marches(gpu, orc, closure, dims, join):  # noqa: F811
    make = lambda p: _case(dims, (closure,), precision=p, join=join, sensor=True)
    ref = _steps(orc, make(abi.PREC_FP64), 2)
    for a, b in zip(ref, _steps(gpu, make(abi.PREC_FP64), 2)):
        assert np.array_equal(a[0], b[0])
    low = _steps(gpu, make(abi.PREC_FP32FLUX), 2)
    for v in (0, -1):
        num = sum(np.abs(a[0][..., v] - b[0][..., v]).sum() for a, b in zip(ref, low))
        assert num <= 1e-5 * sum(np.abs(a[0][..., v]).sum() for a in ref)
