"""Implicit residual smoothing in the FP32-flux form of a coupled run: its stages run in FP64, source included, so
it steps to the plain form's bits, with and without evaporation, in 1-D, 2-D and 3-D."""
import numpy as np
import pytest

from ice_b200 import abi
from test_gpu_faces import _case, _steps, gpu  # noqa: F401

pytestmark = pytest.mark.gpu


def _coupled(dims, evap, precision):
    case = _case(dims, ("IG", "AG"), precision=precision)
    num = case.numerics
    num.time_accurate, num.irs, num.irs_beta, num.coupled, num.cfl = False, True, 0.5, True, 0.2
    num.drag, num.heat = "Schiller-Naumann", "Ranz-Marshall"
    for fam in case.families:
        fam.lv_al, fam.Mv, fam.cpv, fam.Le, fam.Tboil = 2.26e6, 18.015, 1996.0, 1.0, 373.15
        fam.evap = "CEM" if evap else "none"
    full = lambda v: np.full(dims[::-1], float(v))
    case.gas.append({"prim5": np.stack([full(v) for v in (1.2, 8.0, 3.0, -2.0, 400.0)], axis=-1), "R": full(287.05),
                     "gam": full(1.4), "k": full(0.026), "mu": full(1.8e-5)})
    return case


@pytest.mark.parametrize("dims", [(40, 1, 1), (18, 9, 1), (12, 9, 10)], ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("evap", [False, True], ids=["inert", "evaporating"])
def test_irs_source_is_fp64_in_both_forms(gpu, orc, dims, evap):  # noqa: F811
    ref = _steps(orc, _coupled(dims, evap, abi.PREC_FP64))
    for precision in (abi.PREC_FP64, abi.PREC_FP32FLUX):
        got = _steps(gpu, _coupled(dims, evap, precision))
        for u, v in zip(ref[0], got[0]):
            assert np.array_equal(u, v), (precision, np.abs(u - v).max())
