"""Boundary tables that list a face of a cell twice, plain form: every record's flux counts, in the order of the
faces and, on one face, of the table, as the oracle adds them (one thread, so that its ghosts take the table's order
too)."""
import os

import numpy as np
import pytest

from ice_b200 import abi
from test_gpu_faces import _case, _steps, gpu  # noqa: F401

pytestmark = pytest.mark.gpu
DIMS = (10, 9, 7)


def _rows(case, b, f):
    return [n for n, r in enumerate(case.bc_rows) if r[0] == b and r[4] == f]


def _open(case):
    case.bc_rows.append(case.bc_rows[0])
    case.bc_rows.append(case.bc_rows[0])


def _wall_and_open(case):
    b, i, j, k, f, _, _ = case.bc_rows[3]
    case.bc_rows.append((b, i, j, k, f, 300, ()))


def _owner_again(case):                  # the connection's owner: the even face of block 1
    case.bc_rows.append(case.bc_rows[_rows(case, 1, 2)[5]])


def _owner_and_wall(case):
    b, i, j, k, f, _, _ = case.bc_rows[_rows(case, 1, 2)[5]]
    case.bc_rows.append((b, i, j, k, f, 300, ()))


def _partner_and_wall(case):
    b, i, j, k, f, _, _ = case.bc_rows[_rows(case, 2, 1)[7]]
    case.bc_rows.insert(2, (b, i, j, k, f, 300, ()))


@pytest.fixture
def one_thread(orc):
    orc.set_threads(1)
    yield orc
    orc.set_threads(os.cpu_count())


def _pair(gpu, orc, make):
    ref, got = _steps(orc, make()), _steps(gpu, make())
    for a, b in zip(ref, got):
        for u, v in zip(a, b):
            assert np.array_equal(u, v), np.abs(u - v).max()


@pytest.mark.parametrize("edit,join,code", [
    (_open, None, 400), (_open, None, 200), (_wall_and_open, None, 400), (_owner_again, 0, 400),
    (_owner_and_wall, 0, 400), (_partner_and_wall, 0, 400)],
    ids=["open", "symmetry", "wall_and_open", "owner_again", "owner_and_wall", "partner_and_wall"])
def test_every_record_counts_once(gpu, one_thread, edit, join, code):  # noqa: F811
    def make():
        case = _case(DIMS, ("MK", "IG", "AG"), code=code, join=join, sensor=join is not None)
        edit(case)
        return case
    _pair(gpu, one_thread, make)


@pytest.mark.parametrize("dims,row", [((33, 1, 1), 0), ((12, 11, 1), 30)], ids=["1d", "2d"])
def test_forms_agree_on_a_face_listed_twice(gpu, orc, dims, row):  # noqa: F811
    def make(precision):
        case = _case(dims, ("IG",), precision=precision)
        case.bc_rows.append(case.bc_rows[row])
        return case
    ref, got = _steps(orc, make(abi.PREC_FP64)), _steps(gpu, make(abi.PREC_FP32FLUX))
    for v in (0, -1):
        a, b = ref[0][0][..., v], got[0][0][..., v]
        assert np.abs(a - b).sum() <= 1e-5 * np.abs(a).sum()
