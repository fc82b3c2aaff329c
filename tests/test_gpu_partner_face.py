"""A boundary table paired by its caller whose connection records name another face of the partner's cell than the
partner's own record: the flux goes through the partner's face, only the ghosts follow the name, as on the oracle."""
import numpy as np
import pytest

from test_gpu_faces import _case, _steps, gpu  # noqa: F401

pytestmark = pytest.mark.gpu


def test_partner_takes_the_flux_on_its_own_face(gpu, orc):  # noqa: F811
    def make():
        case = _case((10, 9, 7), ("IG", "AG"), join=0)
        case.build_geometry()
        case.build_records(gpu)
        own = (case.rec_int[:, 5] == 101) & (case.rec_int[:, 13] == 1)
        case.rec_int[own, 11] = 5 + (case.rec_int[own, 10] != 1)       # faces 5 and 6 of the partner's cells
        return case
    ref, got = _steps(orc, make()), _steps(gpu, make())
    for a, b in zip(ref, got):
        for u, v in zip(a, b):
            assert np.array_equal(u, v), np.abs(u - v).max()
