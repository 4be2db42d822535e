"""The grouped solution update of single solves whose vectors outgrow L2
(x += alpha p of several iterations at once), at stops inside and at the ends
of a group.  FP64: bit for bit the batched solve of the same case, which
updates x every iteration.  Refined: x after a few iterations is the FP64
one to the FP32 rounding of p (2^-24 per iteration, n of them, and the
directions' own FP32 drift of the same size: 64 n 2^-24 of x's norm)."""
import numpy as np
import pytest

from pot3d_b200 import host
from pot3d_b200.host import PM_R1
from pot3d_b200.solver import BatchSolver, Pot3dSolver

pytestmark = pytest.mark.gpu

DIMS = (131, 150, 260)  # 5.0 M padded unknowns: above both thresholds of the rule


def _case():
    mesh = host.make_mesh(*DIMS)
    tn, pn, fi = host.synthetic_br(4, 15, 4, mesh.nt, mesh.np)
    return mesh, host.br0_from_map(mesh, tn, pn, fi)


def _x(s, b, ncgmax, eps=1e-12):
    x = np.zeros(s.N)
    s.cgsolve(x, b.copy(), ncgmax=ncgmax, epscg=eps)
    return x, s.last_info.ncg


@pytest.fixture(scope="module")
def case():
    return _case()


def test_fp64_groups_bitwise_at_every_stop(cuda, case):
    mesh, br0 = case
    stops = (1, 2, 3, 4, 5, 8, 30, 63, 64, 65)
    with Pot3dSolver(mesh, br0) as s, BatchSolver([mesh], [br0], [PM_R1["ss"]]) as b:
        rhs = s.rhs()
        for n in stops:
            x, ncg = _x(s, rhs, n)
            b.solve(epscg=1e-12, ncgmax=n)
            assert ncg == n == b.infos[0].ncg
            assert np.array_equal(x, b.solution(0)), n


@pytest.mark.parametrize("ifprec", [1, 2])
def test_refined_groups_follow_fp64(cuda, case, ifprec):
    mesh, br0 = case
    with Pot3dSolver(mesh, br0, ifprec=ifprec) as s, \
            Pot3dSolver(mesh, br0, ifprec=ifprec, precision="fp32_refined") as f:
        rhs = s.rhs()
        for n in (1, 7, 8, 9, 13):
            x, _ = _x(s, rhs, n)
            y, ncg = _x(f, rhs, n)
            assert ncg == n
            assert np.linalg.norm(y - x) <= 64 * n * 2.0 ** -24 * np.linalg.norm(x), n
