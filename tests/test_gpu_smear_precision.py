"""Rounding of the Gaussian smearing stencil against sums in extended precision, for every grouping of fields a
thread takes, on grids whose steps overlap their launches (up to 8,192 blocks) and on larger ones (compiled apart).

The bar is the error of an FP64 sum that adds the 18 complex products of a component one after the other, formed
here from the same inputs.  A sum of six partial sums of three products rounds the large running sum a third
as often, so it stays below that; one chain of 36 fused multiply-adds rounds it twice as often and does not.
alpha = 0.5 makes the norm 1 / (1 + 6 alpha) exact.  Over the 49,152 and more numbers compared the two rms errors
are known to better than 1%."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ALPHA = 0.5


def _step(L, U, psi, ctype):
    """One step on the time slices given (U, psi: [T, Z, Y, X, ...]), every product added in turn."""
    u, p = U.astype(ctype), psi.astype(ctype)
    acc = np.zeros_like(p)
    for mu in range(3):
        ax = 3 - mu
        f, ub, g = np.roll(p, -1, ax), np.roll(u[..., mu, :, :], 1, ax), np.roll(p, 1, ax)
        for j in range(3):
            acc = acc + u[..., mu, None, :, j] * f[..., j, None]
        for j in range(3):
            acc = acc + ub[..., None, j, :].conj() * g[..., j, None]
    a = p.real.dtype.type(ALPHA)
    return (p + a * acc) * p.real.dtype.type(0.25)


SMALL, LARGE = ((8, 8, 8, 8), range(8)), ((16, 16, 16, 34), (0, 33))


# SMALL: 128 blocks of 32 sites of both parities a group of fields (up to 256); LARGE: 4,352 (up to 8,704), where six
# fields go to one group of six
@pytest.mark.parametrize("lattice,n", [(SMALL, 1), (SMALL, 3), (SMALL, 4), (SMALL, 6), (LARGE, 2), (LARGE, 5), (LARGE, 6),
                                       (LARGE, 8), (LARGE, 12)])
def test_no_further_off_than_a_plain_sum(qkx, oracle, lattice, n):
    L, slices = lattice
    dims = (L[3], L[2], L[1], L[0])
    U = oracle.gauge_random(L, 0.3, 61)
    Uc = np.ascontiguousarray(U).view(np.complex128).reshape(dims + (4, 3, 3))[list(slices)]
    psis = [oracle.spinor_gaussian(L, 70 + i) for i in range(n)]
    with qkx.Lattice(qkx.LatticeInfo(L=L)) as lat:
        lat.load_smearing_gauge(U)
        outs = lat.Gaussian_smearing(psis, nsmear=1, alpha=ALPHA)
    err = bar = ref = 0.0
    for p, o in zip(psis, outs):
        pc = np.ascontiguousarray(p).view(np.complex128).reshape(dims + (4, 3))[list(slices)]
        oc = np.ascontiguousarray(o).view(np.complex128).reshape(dims + (4, 3))[list(slices)]
        exact = _step(L, Uc, pc, np.clongdouble)
        err += float(np.sum(np.abs(oc - exact) ** 2))
        bar += float(np.sum(np.abs(_step(L, Uc, pc, np.complex128) - exact) ** 2))
        ref += float(np.sum(np.abs(exact) ** 2))
    err, bar = (err / ref) ** 0.5, (bar / ref) ** 0.5
    assert err <= bar, (err, bar)
