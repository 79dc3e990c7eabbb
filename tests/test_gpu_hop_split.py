"""The FP64 hop that splits a site over two threads (hop_s2_kernel) where its grid and batch
rules change: partial last blocks of 32 sites, and two right-hand sides a thread with an odd
batch and a masked right-hand side.  Oracle: the restatement of the reference's operator.
Tolerances: 1e-13 relative for FP64 operators (the bar of the operator tests), the solver's
own 1e-10 for true residuals."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [(2, 2, 2, 4), (2, 4, 2, 4), (4, 2, 6, 6), (10, 6, 2, 14), (34, 2, 4, 6)])
@pytest.mark.parametrize("op", ["tm", "tm_dagtm", "tm_xx_dagtm_xx_oo", "tm_xx_chiral_ee"])
def test_partial_blocks(qkx, oracle, L, op):
    """V/2 = 8 to 408: fewer sites than a block, exact multiples of 32, and remainders."""
    U = oracle.apply_bc(L, oracle.gauge_random(L, 0.3, 31), -1)
    psi = oracle.spinor_gaussian(L, 32)
    with qkx.Lattice(qkx.LatticeInfo(L=L, kappa=0.1615, mu=0.004)) as lat:
        lat.load_gauge(U)
        assert rel(lat.apply(op, psi), oracle.apply(op, L, U, psi, 0.1615, 0.004)) < 1e-13


def test_two_rhs_a_thread(qkx, oracle):
    """1,024 site blocks with a remainder of 24 sites: an odd batch takes two right-hand sides a
    thread, one of them zero (masked from the start)."""
    L, kappa, mu = (10, 14, 18, 26), 0.16, 0.01
    U = oracle.apply_bc(L, oracle.gauge_random(L, 0.3, 41), -1)
    bs = [oracle.spinor_gaussian(L, 50), np.zeros_like(oracle.spinor_gaussian(L, 50)), oracle.spinor_gaussian(L, 51)]
    with qkx.Lattice(qkx.LatticeInfo(L=L, kappa=kappa, mu=mu)) as lat:
        lat.load_gauge(U)
        for prec in (qkx.PREC_HALF, qkx.PREC_DOUBLE):
            xs, info = lat.invert(bs, precision=prec, tol=1e-10)
            assert info.converged and np.all(xs[1] == 0.0)
            worst = 0.0
            for i in (0, 2):
                r = bs[i] - oracle.apply("tm", L, U, xs[i], kappa, mu)
                worst = max(worst, float(np.linalg.norm(r) / np.linalg.norm(bs[i])))
            assert worst <= 1e-10
            assert abs(worst - info.true_residual) <= 1e-3 * worst
