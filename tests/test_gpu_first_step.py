"""A context's work memory (metric rows, face fluxes) is made with its set-up: the first step of the plain form takes no
more device memory than its graph does, far below the 25 MB of rows and 45 MB of fluxes of this box."""
import pytest
import torch

from ice_b200 import abi
from ice_b200.solver import Solver
from test_gpu_faces import _case, gpu  # noqa: F401

pytestmark = pytest.mark.gpu


def test_the_first_step_allocates_no_work_memory(gpu):  # noqa: F811
    warm = Solver(_case((8, 8, 8), ("IG",), precision=abi.PREC_FP64), gpu)
    warm.step(1)
    s = Solver(_case((64, 64, 64), ("IG",), precision=abi.PREC_FP64), gpu)
    before = torch.cuda.mem_get_info()[0]
    s.step(1)
    assert before - torch.cuda.mem_get_info()[0] < 16 << 20
    s.close()
    warm.close()
