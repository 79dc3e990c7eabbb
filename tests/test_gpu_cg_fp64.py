"""The plain FP64 CG queues iterations ahead of the residual it reads: stops at maxIter, and what the profile of
its hops counts."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu
KAPPA, MU = 0.16, 0.01


@pytest.fixture(scope="module")
def setup(qkx, oracle):
    L = (8, 6, 4, 10)
    U = oracle.apply_bc(L, oracle.gauge_random(L, 0.3, 51), -1)
    lat = qkx.Lattice(qkx.LatticeInfo(L=L, kappa=KAPPA, mu=MU, tol=1e-10, maxIter=1000))
    lat.load_gauge(U)
    yield L, U, lat
    lat.close()


@pytest.mark.parametrize("n", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("start", [False, True])
def test_stops_at_max_iter(qkx, oracle, setup, n, start):
    """Exactly n steps of the reference's recurrence, from zero and from a start vector (FP64: 1e-12 relative
    after at most seven steps, as the products' sums are ordered differently)."""
    L, U, lat = setup
    b = oracle.spinor_gaussian(L, 52)
    x0 = oracle.spinor_gaussian(L, 53) if start else np.zeros_like(b)
    lat.set_params(maxIter=n)
    x, info = lat.cg(b, x0)
    want, k, _ = oracle.cg(L, U, b, KAPPA, MU, tol=1e-10, maxIter=n, x0=x0)
    assert info.iterations == n == k and info.converged == 0
    assert rel(x, want) < 1e-12
    lat.set_params(maxIter=1000)
    x, info = lat.cg(b)
    assert info.converged == 1 and rel(oracle.apply("tm_dagtm", L, U, x, KAPPA, MU), b) < 1.01e-10


def test_profile_counts_the_hops_of_the_iterations_only(qkx, oracle, setup):
    L, U, lat = setup
    b = oracle.spinor_gaussian(L, 54)
    _, plain = lat.cg(b)
    lat.profile_reset()
    lat.profile(True)
    try:
        x, info = lat.cg(b)
    finally:
        lat.profile(False)
    n, _, by = lat.profile_read()
    assert info.iterations == plain.iterations and n == 2 * info.iterations
    V = b.size // 24
    # a hop reads the field and the links and writes a field; the second also reads the residual it updates
    assert by == info.iterations * V * (2 * (2 * 192.0 + 4 * 144.0) + 192.0)


def test_work_fields_that_nothing_reads_are_not_held(qkx, oracle):
    """An operator, a CG and a solve of 16^3 x 32 (24 MiB a field) hold seven work fields."""
    import torch

    def run(L):
        lat = qkx.Lattice(qkx.LatticeInfo(L=L, kappa=KAPPA, mu=MU, maxIter=1000))
        lat.generate_gauge(0.3, 5)
        b, x = lat.field(oracle.spinor_gaussian(L, 55)), lat.field()
        lat.sync()
        free = torch.cuda.mem_get_info()[0]
        lat.apply_dev("tm_xx_dagtm_xx_ee", b, x)
        info = qkx.SolveInfo()
        x.upload(np.zeros((lat.V, 4, 3, 2)))
        qkx.check(qkx.lib().qkx_cg_dev(lat.ctx, b.ptr, x.ptr, C.byref(info)))
        lat.invert_dev([b], [x], method=qkx.SOLVER_CG_FP64, tol=1e-8)
        used = free - torch.cuda.mem_get_info()[0]
        b.close(), x.close(), lat.close()
        return used

    run((4, 4, 4, 8))  # loads every kernel
    L = (16, 16, 16, 32)
    field = 16 * 16 * 16 * 32 * 192
    assert run(L) < 7.5 * field


def test_cg_on_the_tiled_hop(qkx, oracle, monkeypatch):
    """QKX_FP64_TILED=1: the first hop of an iteration on TMA row tiles, with its norm and the mask of queued
    iterations, the second on the direct kernel; same steps, FP64 rounding apart."""
    L = (16, 8, 4, 8)
    U = oracle.apply_bc(L, oracle.gauge_random(L, 0.3, 57), -1)
    b = oracle.spinor_gaussian(L, 58)
    out = []
    for mode in ("0", "1"):
        monkeypatch.setenv("QKX_FP64_TILED", mode)
        with qkx.Lattice(qkx.LatticeInfo(L=L, kappa=KAPPA, mu=MU, tol=1e-10, maxIter=1000)) as lat:
            lat.load_gauge(U)
            out.append(lat.cg(b))
    (x, i), (y, j) = out
    assert i.converged == j.converged == 1 and i.iterations == j.iterations
    assert rel(y, x) < 1e-9
