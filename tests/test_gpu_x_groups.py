"""The grouped solution update of single solves whose vectors outgrow L2
(x += alpha p of several iterations at once), at stops inside and at the ends
of a group.  FP64: bit for bit the batched solve of the same case, which
updates x every iteration.  Refined: x after a few iterations is the FP64
one to the FP32 rounding of p (2^-24 per iteration, n of them, and the
directions' own FP32 drift of the same size: 64 n 2^-24 of x's norm).  The
directions pass through vectors the handle has anyway: what other calls leave
in them changes no bit, and no memory is taken for them."""
import threading

import numpy as np
import pytest

from pot3d_b200 import host
from pot3d_b200.host import PM_R1
from pot3d_b200.solver import BatchSolver, Pot3dSolver

pytestmark = pytest.mark.gpu

NR, NT = 131, 150  # 129 radial points in rows of 144: 15 pad lanes
NRP = 144


def _case():
    """A grid a quarter above the larger threshold of the rule (28 bytes a padded unknown against L2)."""
    import torch
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    mesh = host.make_mesh(NR, NT, 2 + int(1.25 * l2 / 28 / (NRP * (NT - 2))))
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
        assert s.update_group() == 4
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
        assert f.update_group() == 8 and s.update_group() == (4 if ifprec == 1 else 1)
        rhs = s.rhs()
        for n in (1, 7, 8, 9, 13):
            x, _ = _x(s, rhs, n)
            y, ncg = _x(f, rhs, n)
            assert ncg == n
            assert np.linalg.norm(y - x) <= 64 * n * 2.0 ** -24 * np.linalg.norm(x), n


def test_kernel_times_count_the_bytes_of_groups(cuda, case):
    mesh, br0 = case
    with Pot3dSolver(mesh, br0) as s:
        ms, by = s.time_kernels(5)
        assert np.all(ms > 0) and by[0] == 32.0 * s.N and by[1] == 36.0 * s.N
        x, _ = _x(s, s.rhs(), 5)  # and leaves the handle as it was
    with Pot3dSolver(mesh, br0) as s:
        assert np.array_equal(x, _x(s, s.rhs(), 5)[0])


def test_grids_within_l2_update_every_iteration(cuda):
    mesh = host.make_mesh(33, 41, 65)
    br0 = host.br0_from_map(mesh, *host.synthetic_br(4, 15, 4, mesh.nt, mesh.np))
    for precision in ("fp64", "fp32_refined"):
        with Pot3dSolver(mesh, br0, precision=precision) as s:
            assert s.update_group() == 1


@pytest.mark.parametrize("ifprec,precision", [(1, "fp64"), (1, "fp32_refined"), (2, "fp32_refined")])
def test_what_other_calls_leave_in_the_directions(cuda, case, ifprec, precision):
    import torch
    mesh, br0 = case
    with Pot3dSolver(mesh, br0, ifprec=ifprec, precision=precision) as s:
        rhs = s.rhs()
        ref, _ = _x(s, rhs, 13)
        noise = np.random.default_rng(5).standard_normal(s.N) * 10.0 ** np.random.default_rng(6).uniform(-300, 300, s.N)

        def again(what):
            assert np.array_equal(_x(s, rhs, 13)[0], ref), what
            xd, rd = torch.zeros(s.N, dtype=torch.float64, device=cuda), torch.from_numpy(rhs).cuda()
            s.cgsolve_dev(xd, rd, ncgmax=13, epscg=1e-12)
            assert np.array_equal(xd.cpu().numpy(), ref), what

        again("a solve")
        s.finalize_phi(noise)
        again("phi of noise")
        y = torch.empty(s.N, dtype=torch.float64, device=cuda)
        s.ax_dev(torch.from_numpy(noise).cuda(), y)
        again("an operator application to noise")
        if precision != "fp64":  # FP64 iterations after a stagnation
            s.set_refine(refine_ratio=0.999, stall_drop=1e-300, stall_limit=1)
            _x(s, rhs, 400)
            assert s.refine_info()[1] > 0
            s.set_refine()
            again("a fallback")
        got = {}
        t = threading.Thread(target=lambda: got.update(b=[s.rhs() for _ in range(8)]))
        t.start()
        again("calls of another thread")
        t.join()
        assert all(np.array_equal(b, rhs) for b in got["b"])


@pytest.mark.parametrize("ifprec,precision,per_padded", [(1, "fp64", 60), (1, "fp32_refined", 76)])
def test_directions_take_no_memory(cuda, ifprec, precision, per_padded):
    """Seven FP64 vectors, a_i and (refined) four FP32 ones, padded, and two
    packed vectors of staging; the rotation's would be 16 or 24 bytes more."""
    import torch
    mesh = host.make_mesh(255, 181, 361)
    br0 = np.asfortranarray(np.cos(mesh.th)[:, None] * np.ones(mesh.np)[None, :])
    free = []
    for _ in range(2):  # the first creation loads the kernels
        before = torch.cuda.mem_get_info()[0]
        with Pot3dSolver(mesh, br0, ifprec=ifprec, precision=precision) as s:
            assert s.update_group() > 1
            free.append(before - torch.cuda.mem_get_info()[0])
            N = s.N
    padded = 256 * 179 * 359
    slack = (8 << 20) + 16 * (2 << 20) + (8 << 20)  # history, 2 MB granules of the vectors, small arrays
    assert free[1] <= per_padded * padded + 16 * N + slack
