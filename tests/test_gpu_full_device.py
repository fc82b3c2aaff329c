"""Calls that take device memory for the first time after the stepping has begun, on a device whose rest another
program holds: they fit where they fitted without the face fluxes and metric rows, which then go to host memory, and the
steps keep their bits."""
import numpy as np
import pytest
import torch

from ice_b200 import abi
from test_gpu_faces import _case, gpu  # noqa: F401
from ice_b200.solver import Solver

pytestmark = pytest.mark.gpu
DIMS = (96, 96, 96)                  # AG: 96 MB of staging for step_host, 85 MB of imports, 340 MB of rows and fluxes
LEFT = 64 << 20


def _fill():
    """Tensors that leave LEFT bytes of the device."""
    torch.cuda.empty_cache()
    held = []
    for chunk in (1 << 30, 16 << 20):
        while torch.cuda.mem_get_info()[0] > LEFT + chunk:
            held.append(torch.empty(chunk, dtype=torch.uint8, device="cuda"))
    return held


def _run(gpu, full, call):
    case = _case(DIMS, ("AG",), precision=abi.PREC_FP64)
    warm = _case((8, 8, 8), ("AG",), precision=abi.PREC_FP64)          # the kernels' own memory, before the device is full
    held = []
    for c in (warm, case):
        s = Solver(c, gpu)
        s.step(1)
        if c is case and full:
            held = _fill()
        try:
            if call == "step_host":
                src = [[a.copy() for a in per] for per in s.download_all()]
                s.step_host(src, src, 1)
                s.step(1)
            else:
                imp = np.zeros((*c.dims[0][::-1], 12))
                imp[..., 0] = 1e-6
                s._check(gpu.set_imports(s.ctx, 1, 1, abi.ptr(imp)), "set_imports")
                s.step(2)
            got = s.download(0, 0)[2:-2, 2:-2, 2:-2]
        finally:
            del held
            held = []
            torch.cuda.empty_cache()
            s.close()
    return got


@pytest.mark.parametrize("call", ["step_host", "set_imports"])
def test_what_fitted_still_fits(gpu, call):  # noqa: F811
    assert np.array_equal(_run(gpu, False, call), _run(gpu, True, call))
