"""The flux and cell kernels at the sizes where their indexing can go wrong: rows around the 31 faces of a warp and
the 124 cells of a CTA, columns around a march's length and around the 128 threads of a CTA, blocks of one and
two cells along a direction, every boundary code, joined blocks, families of which one has a face flux and
another none, a face listed twice. The plain form steps to the oracle's bits; the FP32-flux form stays within
1e-5 of it (relative L1 of the density and the number density: some 50 roundings of 6e-8 on each flux, half of
which a CFL of 0.5 moves into a cell, over three stages)."""
import numpy as np
import pytest

from ice_b200 import abi, configs
from ice_b200.case import Case, Family, Numerics, box_bc, box_nodes, empty_state
from ice_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from ice_b200 import build
    build.build()
    return abi.load_gpu()


def _case(dims, closures=("IG",), code=400, limiter="vanleer", precision=0, riemann="", sensor=False, join=None,
          twice=False):
    """A box of dims cells with a smooth stream; join: cut in two blocks along that axis."""
    h = 1e-3
    spans = [(0, dims[join or 0])] if join is None else [(0, dims[join] // 2), (dims[join] // 2, dims[join])]
    d = join or 0
    blocks = [tuple(hi - lo if a == d else dims[a] for a in range(3)) for lo, hi in spans]
    nodes = [box_nodes(*bd, lo=tuple(lo * h if a == d else 0.0 for a in range(3)), size=tuple(q * h for q in bd))
             for (lo, hi), bd in zip(spans, blocks)]
    rows = []
    for b, bd in enumerate(blocks):
        codes = {f: (0 if dims[(f - 1) // 2] == 1 and code != 200 else code) for f in range(1, 7)}
        if join is not None:
            codes[2 * d + 2 - b] = 101
        for row in box_bc(b + 1, bd, codes):
            bb, i, j, k, f, c, pay = row
            if c == 101:
                src = [i, j, k]
                src[d] = 1 if b == 0 else blocks[0][d]
                row = (bb, i, j, k, f, 101, (2 - b, *src, f - 1 if f % 2 == 0 else f + 1))
            rows.append(row)
    if twice:
        rows.append(rows[0])
    fams = [Family(cl, riemann=riemann if cl != "MK" else "", rho_al=1000.0, cs_al=4180.0) for cl in closures]
    num = Numerics(scheme="RK3", cfl=0.5, dt_max=1.0, limiter=limiter, shock_detector=sensor, precision=precision)
    case = Case("faces", nodes, fams, num, rows)
    rng = np.random.default_rng(3)
    ph = rng.uniform(0, 6.28, size=3)
    for (lo, hi), bd in zip(spans, blocks):
        x, y, z = (np.arange(bd[a]) + (lo if a == d else 0) for a in range(3))
        wave = (np.cos(0.3 * x + ph[0])[None, None, :] * np.cos(0.23 * y + ph[1])[None, :, None]
                * np.cos(0.37 * z + ph[2])[:, None, None])
        per = []
        for fam in fams:
            st = empty_state(bd, fam.nc)
            I = st[2:-2, 2:-2, 2:-2]
            I[...] = 0.0
            rho = 1e-3 * (1.0 + 0.4 * wave)
            I[..., 0], I[..., 1], I[..., 2], I[..., 3] = rho, 3.0 + wave, -2.0 * wave, 1.0 - 0.5 * wave
            for q in {"MK": (), "IG": (4,), "AG": (4, 7, 9)}[fam.closure]:
                I[..., q] = rho * (1.0 + 0.1 * q)
            if fam.closure == "AG":
                I[..., 5] = 0.2 * rho
            I[..., -2], I[..., -1] = 300.0 + 20.0 * wave, rho / 4e-12
            per.append(st)
        case.state.append(per)
    return case


def _steps(lib, case, n=3):
    s = Solver(case, lib)
    out = s.step(n)
    assert out.status == 0
    got = [[q[2:-2, 2:-2, 2:-2] for q in per] for per in s.download_all()]
    s.close()
    return got


SIZES = [(31, 1, 1), (32, 1, 1), (33, 5, 1), (124, 3, 1), (125, 2, 2), (2, 2, 2), (1, 40, 3), (3, 1, 40), (17, 18, 17),
         (16, 129, 4), (64, 3, 33), (5, 30, 31)]


@pytest.mark.parametrize("dims", SIZES, ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("closure", ["MK", "IG", "AG"])
def test_sizes(gpu, orc, dims, closure):
    ref = _steps(orc, _case(dims, (closure,)))
    for u, v in zip(ref[0], _steps(gpu, _case(dims, (closure,)))[0]):
        assert np.array_equal(u, v)
    got = _steps(gpu, _case(dims, (closure,), precision=abi.PREC_FP32FLUX))
    for v in (0, -1):
        a, b = ref[0][0][..., v], got[0][0][..., v]
        assert np.abs(a - b).sum() <= 1e-5 * np.abs(a).sum()


@pytest.mark.parametrize("kw", [dict(limiter=q) for q in abi.LIMITER] +
                         [dict(code=c, sensor=c == 300) for c in (200, 300, 301)] +
                         [dict(join=d, sensor=True) for d in (0, 1, 2)] + [dict(riemann="HLLE"), dict(twice=True)],
                         ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()))
def test_forms(gpu, orc, kw):
    make = lambda p: _case((18, 9, 7), ("MK", "IG", "AG"), precision=p, **kw)
    ref, got = _steps(orc, make(0)), _steps(gpu, make(0))
    for p in range(3):
        for a, b in zip(ref, got):
            assert np.array_equal(a[p], b[p]) if not kw.get("twice") else np.allclose(a[p], b[p], rtol=1e-12, atol=0.0)
    low = _steps(gpu, make(abi.PREC_FP32FLUX))
    for p in range(3):
        for v in (0, -1):
            num = sum(np.abs(a[p][..., v] - b[p][..., v]).sum() for a, b in zip(ref, low))
            assert num <= 1e-5 * sum(np.abs(a[p][..., v]).sum() for a in ref)
