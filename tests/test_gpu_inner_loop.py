"""The mixed solver's inner loop as one cooperative kernel: which batches take it (at most 592 items of 32 sites and
one right-hand side, alone on the GPU), several blocks an SM, masked right-hand sides, its barrier's limit,
and solves beside each other.  A solve whose iterations are launched kernel by kernel counts more than eight launches
an iteration; with one kernel for the inner loop it counts only those around it."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KAPPA, MU, TOL = 0.16, 0.01, 1e-10


def _lattice(qkx, oracle, L, seed=81):
    U = oracle.apply_bc(L, oracle.gauge_random(L, 0.3, seed), -1)
    lat = qkx.Lattice(qkx.LatticeInfo(L=L, kappa=KAPPA, mu=MU))
    lat.load_gauge(U)
    return lat, U


def _res(O, L, U, x, b):
    return float(np.linalg.norm(b - O.apply("tm", L, U, x, KAPPA, MU)) / np.linalg.norm(b))


def _solve(lat, bs, **kw):
    k = lat.kernel_launches()
    xs, info = lat.invert(bs, tol=TOL, **kw)
    return xs, info, lat.kernel_launches() - k


def _one_kernel(info, launches):
    return launches < 4 * info.iterations


# items: 297, 384, 473, 512, 592 (the last that the rule takes), 594
@pytest.mark.parametrize("prec", ["half", "single"])
@pytest.mark.parametrize("L,n,inside", [((22, 6, 12, 12), 1, True), ((8, 8, 8, 16), 3, True),
                                        ((12, 14, 10, 18), 1, True), ((8, 8, 8, 16), 4, True),
                                        ((4, 4, 8, 74), 4, True), ((22, 6, 12, 12), 2, False)])
def test_rule_and_host_loop_bits(qkx, oracle, L, n, inside, prec):
    p = {"half": qkx.PREC_HALF, "single": qkx.PREC_SINGLE}[prec]
    lat, U = _lattice(qkx, oracle, L)
    with lat:
        bs = [oracle.spinor_gaussian(L, 82 + i) for i in range(n)]
        if n > 2:
            bs[1] = np.zeros_like(bs[1])  # masked from the start
        xs, info, k = _solve(lat, bs, precision=p)
        assert _one_kernel(info, k) == inside
        host, ih, kh = _solve(lat, bs, precision=p, use_graphs=0)
        assert not _one_kernel(ih, kh)
        assert (info.iterations, info.reliable_updates, info.restarts) == (ih.iterations, ih.reliable_updates, ih.restarts)
        for b, x, y in zip(bs, xs, host):
            assert np.array_equal(x, y)
            assert _res(oracle, L, U, x, b) <= TOL if np.any(b) else not np.any(x)


@pytest.mark.parametrize("L,n", [((8, 8, 8, 16), 1), ((8, 8, 8, 16), 3)])
@pytest.mark.parametrize("prec", ["half", "single"])
def test_barrier_that_gives_up_leaves_the_solve_to_the_kernels(qkx, oracle, monkeypatch, L, n, prec):
    """With no time to wait the blocks give up at their first barrier; the solve then runs kernel by kernel
    from the start and has the bits of the host-driven loop, again and again on the same context, the
    solution field being the source's own as well."""
    p = {"half": qkx.PREC_HALF, "single": qkx.PREC_SINGLE}[prec]
    monkeypatch.setenv("QKX_INNER_WAIT_MS", "0")
    lat, U = _lattice(qkx, oracle, L)
    monkeypatch.delenv("QKX_INNER_WAIT_MS")
    with lat:
        bs = [oracle.spinor_gaussian(L, 82 + i) for i in range(n)]
        host, ih, _ = _solve(lat, bs, precision=p, use_graphs=0)
        for _ in range(2):
            xs, info, k = _solve(lat, bs, precision=p)
            assert info.converged == 1 and info.iterations == ih.iterations and not _one_kernel(info, k)
            for b, x, y in zip(bs, xs, host):
                assert np.array_equal(x, y) and _res(oracle, L, U, x, b) <= TOL
        f = [lat.field(b) for b in bs]
        assert lat.invert_dev(f, f, precision=p, tol=TOL).converged == 1
        for q, y in zip(f, host):
            assert np.array_equal(q.download(), y)
            q.close()


def test_two_solves_at_once(qkx, oracle):
    """Two threads, two lattices, solve after solve: the cooperative grids take turns or share the GPU, and every
    solution has the bits of the same solve alone."""
    specs = [((8, 8, 8, 16), 4), ((12, 14, 10, 18), 1)]
    lats = [_lattice(qkx, oracle, L, 90 + i) for i, (L, _) in enumerate(specs)]
    bs = [[oracle.spinor_gaussian(L, 91 + 7 * i + r) for r in range(n)] for i, (L, n) in enumerate(specs)]
    alone = [lat.invert(b, tol=TOL)[0] for (lat, _), b in zip(lats, bs)]
    bad = []

    def work(i):
        try:
            for _ in range(20):
                xs, info = lats[i][0].invert(bs[i], tol=TOL)
                if info.converged != 1 or not all(np.array_equal(x, y) for x, y in zip(xs, alone[i])):
                    bad.append(i)
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for lat, _ in lats:
        lat.close()
    assert not bad


def test_a_batch_of_lattices_is_not_alone(qkx, oracle):
    """invert_batch's path with a thread per lattice (here: one lattice's hops are being timed) takes no
    cooperative loop either: its lattices share the GPU."""
    specs = [((8, 8, 8, 16), 2), ((6, 4, 2, 10), 3)]
    lats = [_lattice(qkx, oracle, L, 95 + i) for i, (L, _) in enumerate(specs)]
    bs = [[oracle.spinor_gaussian(L, 96 + 7 * i + r) for r in range(n)] for i, (L, n) in enumerate(specs)]
    jobs = [(lat, [lat.field(b) for b in v], [lat.field() for _ in v], [MU] * len(v)) for (lat, _), v in zip(lats, bs)]
    lats[1][0].profile(True)
    k = [lat.kernel_launches() for lat, _ in lats]
    res = qkx.invert_batch(jobs, tol=TOL)
    lats[1][0].profile(False)
    for (lat, U), job, v, r, k0, (L, _) in zip(lats, jobs, bs, res, k, specs):
        assert r["status"] == qkx.OK and lat.kernel_launches() - k0 > 4 * r["info"]["iterations"]
        for x, b in zip(job[2], v):
            assert _res(oracle, L, U, x.download(), b) <= TOL
        for f in job[1] + job[2]:
            f.close()
        lat.close()


@pytest.mark.parametrize("prec", ["half", "single"])
@pytest.mark.parametrize("L,n", [((4, 4, 4, 8), 1), ((8, 8, 8, 16), 1), ((8, 8, 8, 16), 3), ((12, 14, 10, 18), 1),
                                 ((8, 8, 8, 16), 4), ((22, 6, 12, 12), 1)])
def test_tuning_keeps_the_one_kernel_loop(qkx, oracle, L, n, prec):
    """qkx_tune times hops one by one: whichever tile it picks, a small batch alone on the GPU keeps its one-kernel
    loop.  A tile set by hand is taken."""
    p = {"half": qkx.PREC_HALF, "single": qkx.PREC_SINGLE}[prec]
    lat, U = _lattice(qkx, oracle, L)
    with lat:
        bs = [oracle.spinor_gaussian(L, 82 + i) for i in range(n)]
        xs, info, k = _solve(lat, bs, precision=p)
        assert _one_kernel(info, k)
        lat.tune(p, n)
        again, it, kt = _solve(lat, bs, precision=p)
        assert _one_kernel(it, kt) and all(np.array_equal(x, y) for x, y in zip(xs, again))
        lat.set_tile(p, n, (1, 64, 0))
        _, it, kt = _solve(lat, bs, precision=p)
        assert not _one_kernel(it, kt)
        lat.set_tile(p, n, (1, 128, 12))
        again, it, kt = _solve(lat, bs, precision=p)
        assert _one_kernel(it, kt) and all(np.array_equal(x, y) for x, y in zip(xs, again))
