"""Small lattices: the hop that splits a site over four threads by direction (tile kind 12) and the
inner loop as one cooperative kernel, at the sizes where they can go wrong: partial blocks of 32 sites,
more items than fit the GPU at once, masked right-hand sides, maxIter inside the loop.  The operator is
checked with the tolerances of the other tiles, solutions by the oracle's residual, and the device loop
against the host-driven one bit for bit (the same kernels' arithmetic in the same order)."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


def _res(O, L, U, x, b, kappa, mu):
    r = b - O.apply("tm", L, U, x, kappa, mu)
    return float(np.linalg.norm(r) / np.linalg.norm(b))


@pytest.mark.parametrize("prec,tol", [("half", 1e-2), ("single", 1e-5)])
@pytest.mark.parametrize("L,n", [((2, 2, 2, 4), 1), ((6, 4, 2, 10), 3), ((4, 4, 4, 8), 2)])
def test_operator_split_by_direction(qkx, oracle, L, n, prec, tol):
    U = oracle.apply_bc(L, oracle.gauge_random(L, 0.3, 71), -1)
    bs = [oracle.spinor_gaussian(L, 72 + i) for i in range(n)]
    p = {"half": qkx.PREC_HALF, "single": qkx.PREC_SINGLE}[prec]
    with qkx.Lattice(qkx.LatticeInfo(L=L, kappa=0.1615, mu=0.004)) as lat:
        lat.load_gauge(U)
        for b, g in zip(bs, lat.sloppy_normal(bs, p, (1, 128, 12))):
            assert rel(g, oracle.apply("tm_xx_dagtm_xx_ee", L, U, b, 0.1615, 0.004)) < tol
        with pytest.raises(qkx.QkxError):
            lat.sloppy_normal(bs, qkx.PREC_DOUBLE, (1, 128, 12))


# 1 to 8 x 128 items (8^3x16), 8 to 15 partial blocks, and 1,185 items (above the rule: kernel by kernel)
@pytest.mark.parametrize("prec", ["half", "single"])
@pytest.mark.parametrize("L,n", [((8, 8, 8, 16), 1), ((8, 8, 8, 16), 5), ((6, 4, 2, 10), 3), ((12, 14, 10, 18), 2),
                                 ((12, 14, 10, 18), 3)])
def test_device_loop_and_host_loop_agree_bitwise(qkx, oracle, L, n, prec):
    kappa, mu = 0.16, 0.01
    U = oracle.apply_bc(L, oracle.gauge_random(L, 0.3, 81), -1)
    bs = [oracle.spinor_gaussian(L, 82 + i) for i in range(n)]
    if n > 2:
        bs[1] = np.zeros_like(bs[1])  # masked from the start
    p = {"half": qkx.PREC_HALF, "single": qkx.PREC_SINGLE}[prec]
    with qkx.Lattice(qkx.LatticeInfo(L=L, kappa=kappa, mu=mu)) as lat:
        lat.load_gauge(U)
        xs, info = lat.invert(bs, precision=p, tol=1e-10)
        again, _ = lat.invert(bs, precision=p, tol=1e-10)
        host, ih = lat.invert(bs, precision=p, tol=1e-10, use_graphs=0)
        assert (info.iterations, info.reliable_updates, info.restarts) == (ih.iterations, ih.reliable_updates, ih.restarts)
        for b, x, y, z in zip(bs, xs, again, host):
            assert np.array_equal(x, y) and np.array_equal(x, z)
            if np.any(b):
                assert _res(oracle, L, U, x, b, kappa, mu) <= 1e-10
            else:
                assert not np.any(x)
        # maxIter inside the inner loop: stops there, says so, and leaves the solver usable
        with pytest.raises(qkx.QkxError) as e:
            lat.invert(bs, precision=p, tol=1e-10, maxIter=3)
        assert e.value.code == qkx.ERR_NOT_CONVERGED
        last, _ = lat.invert(bs, precision=p, tol=1e-10)
        assert all(np.array_equal(x, y) for x, y in zip(xs, last))


@pytest.mark.parametrize("L,n", [((2, 2, 2, 2), 1), ((6, 4, 2, 10), 3), ((8, 8, 8, 16), 5)])
@pytest.mark.parametrize("nt", [64, 128, 256])
def test_fp32_one_rhs_a_thread(qkx, oracle, L, n, nt):
    """The FP32 hop that loads a term ahead: extents of 2 (both neighbours are one site), partial blocks, and
    a solve in which one right-hand side is masked from the start."""
    kappa, mu = 0.16, 0.01
    U = oracle.apply_bc(L, oracle.gauge_random(L, 0.3, 91), -1)
    bs = [oracle.spinor_gaussian(L, 92 + i) for i in range(n)]
    with qkx.Lattice(qkx.LatticeInfo(L=L, kappa=kappa, mu=mu)) as lat:
        lat.load_gauge(U)
        for b, g in zip(bs, lat.sloppy_normal(bs, qkx.PREC_SINGLE, (1, nt, 0))):
            assert rel(g, oracle.apply("tm_xx_dagtm_xx_ee", L, U, b, kappa, mu)) < 1e-5
        if n == 1:
            return
        lat.set_tile(qkx.PREC_SINGLE, n, (1, nt, 0))
        bs[0] = np.zeros_like(bs[0])
        xs, _ = lat.invert(bs, precision=qkx.PREC_SINGLE, tol=1e-10)
        assert not np.any(xs[0])
        for b, x in zip(bs[1:], xs[1:]):
            assert _res(oracle, L, U, x, b, kappa, mu) <= 1e-10
