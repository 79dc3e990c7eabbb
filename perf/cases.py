"""The work a user of qkxtm_mpi_b200 has it do, as cases that can be timed and checked.

Kinds of case (``case["kind"]``):

* ``op``     one application of a twisted-mass operator to a device field (``Lattice.apply_dev``)
* ``blas``   the vector work of one CG iteration (``reCdotXdagY``, ``X_eq_X_p_aY``, ``norm2``, ``X_eq_aX_p_Y``)
* ``solve``  ``Lattice.invert_dev`` on device fields: the even-odd mixed-precision CG for a batch of
             right-hand sides, or the plain FP64 CG
* ``batch``  ``invert_batch``: solves on several lattices of different sizes in one call
* ``smear``  ``Lattice.Gaussian_smearing_dev`` of a batch of fields with its smearing links
* ``twopt``  ``Lattice.meson_2pt`` for all ten operators and ``Lattice.nucleon_2pt``, from device propagators

Lattices, masses, link smoothness (U = exp(i eps H)) and batch sizes are those of this repository's tests and
benchmark (8^3x16 to 32^3x64, kappa 0.1615, mu 0.0015 to 0.01, 1 to 12 right-hand sides) and generic ones between
them.  Device fields are torch tensors in the library's even-odd layout [parity][spin*3+colour][V/2].

``exact`` states every result in torch complex128 from the definitions: the Wilson hopping term by shifts of the
whole lattice, the operators from it, solutions by a complex128 CG run to rounding, correlators by tensor sums.
"""
import math

import torch

import qkxtm_mpi_b200 as qkx

DEV = "cuda"
C128 = torch.complex128
KAPPA = 0.1615
PREC = {"half": qkx.PREC_HALF, "single": qkx.PREC_SINGLE, "double": qkx.PREC_DOUBLE}
OPS = ["tm", "tm_dag", "tm_dagtm", "wilson", "dslash", "tm_xx_ee", "tm_xx_oo", "tm_xx_dagtm_xx_ee",
       "tm_xx_dagtm_xx_oo", "tm_chiral", "tm_xx_chiral_ee", "tm_xx_dagtm_xx_chiral_oo"]


def _case(kind, L, **kw):
    return {"kind": kind, "lx": L[0], "ly": L[1], "lz": L[2], "lt": L[3], **kw}


def listed():
    return [
        # the operator on the smallest lattice of the tests: what a call costs when the GPU is hardly used
        dict(_case("op", (8, 8, 8, 16), op="tm", mu=0.004), name="tm_8x16"),
        # a lattice with no power of two in it, the other basis, the odd-odd normal operator
        dict(_case("op", (12, 14, 10, 18), op="tm_xx_dagtm_xx_chiral_oo", mu=0.004), name="schur_chiral_ragged"),
        # the Schur normal operator of the even-odd CG at the size of the first production configuration
        dict(_case("op", (24, 24, 24, 48), op="tm_xx_dagtm_xx_ee", mu=0.004), name="schur_24x48"),
        # the full normal operator at the headline lattice: the largest single-field operator
        dict(_case("op", (32, 32, 32, 64), op="tm_dagtm", mu=0.0015), name="tm_dagtm_32x64"),
        # the vector work of a CG that a user's program writes itself on the qkxTM BLAS
        dict(_case("blas", (24, 24, 24, 48)), name="blas_24x48"),
        # the reference's own algorithm, plain FP64 CG, one source
        dict(_case("solve", (16, 16, 16, 32), method="fp64", precision="double", nrhs=1, mu=0.004, tol=1e-10,
                   source="gauss"), name="cg_fp64_16x32"),
        # one source on a small lattice with the default solver: launches and latency
        dict(_case("solve", (8, 8, 8, 16), method="mixed", precision="half", nrhs=1, mu=0.01, tol=1e-10,
                   source="gauss"), name="solve_half_8x16_1"),
        # FP32 sloppy fields, an odd batch, the tightest tolerance of the tests
        dict(_case("solve", (24, 24, 24, 48), method="mixed", precision="single", nrhs=5, mu=0.004, tol=1e-12,
                   source="gauss"), name="solve_single_24x48_5"),
        # the headline: the 12 spin-colour point sources of a propagator at 32^3x64 with FP16 sloppy fields
        dict(_case("solve", (32, 32, 32, 64), method="mixed", precision="half", nrhs=12, mu=0.0015, tol=1e-10,
                   source="point"), name="solve_half_32x64_12"),
        # uneven instances in one call: an ensemble analysis with several volumes
        dict(_case("batch", (16, 16, 16, 32), nrhs=3, mu=0.004, tol=1e-10), name="batch_uneven"),
        # sink smearing of a propagator's 12 columns
        dict(_case("smear", (24, 24, 24, 48), nrhs=12, nsmear=20), name="smear_24x48_12"),
        # two-point functions of a propagator pair with the 33 momenta up to Q^2 = 4
        dict(_case("twopt", (24, 24, 24, 48), qsq=4), name="twopt_24x48"),
    ]


def _extent(rng, lo, hi):
    """An even extent in [lo, hi], spread over its logarithm."""
    return 2 * max(lo // 2, min(hi // 2, round(0.5 * math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _lattice(rng, lo, hi, vmax):
    while True:
        L = (_extent(rng, lo, hi), _extent(rng, lo, hi), _extent(rng, lo, hi), _extent(rng, lo, 2 * hi))
        if 512 <= L[0] * L[1] * L[2] * L[3] <= vmax:
            return L


def draw(rng):
    kind = rng.choice(["op", "op", "op", "blas", "solve", "solve", "solve", "batch", "smear", "twopt"])
    mu = rng.choice([0.0015, 0.004, 0.01])
    if kind == "op":
        return _case("op", _lattice(rng, 4, 32, 32**3 * 64), op=rng.choice(OPS), mu=mu)
    if kind == "blas":
        return _case("blas", _lattice(rng, 4, 32, 32**3 * 64))
    if kind == "solve":
        method = rng.choice(["mixed", "mixed", "mixed", "fp64"])
        if method == "fp64":
            return _case("solve", _lattice(rng, 6, 20, 16**3 * 32), method="fp64", precision="double",
                         nrhs=rng.randint(1, 2), mu=0.004, tol=rng.choice([1e-10, 1e-12]), source="gauss")
        return _case("solve", _lattice(rng, 6, 24, 24**3 * 48), method="mixed",
                     precision=rng.choice(["half", "half", "single"]), nrhs=rng.randint(1, 12),
                     mu=rng.choice([0.004, 0.01]), tol=rng.choice([1e-10, 1e-12]),
                     source=rng.choice(["gauss", "point"]))
    if kind == "batch":
        return _case("batch", _lattice(rng, 8, 16, 16**3 * 32), nrhs=rng.randint(1, 6), mu=mu, tol=1e-10)
    if kind == "smear":
        return _case("smear", _lattice(rng, 4, 24, 24**3 * 48), nrhs=rng.randint(1, 12), nsmear=rng.randint(1, 20))
    return _case("twopt", _lattice(rng, 4, 24, 24**3 * 48), qsq=rng.randint(0, 4))


# ------------------------------------------------------------------ inputs
def _dims(case):
    return (case["lx"], case["ly"], case["lz"], case["lt"])


def _volume(L):
    return L[0] * L[1] * L[2] * L[3]


def _rng(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _normal(shape, g):
    """Complex normals of unit variance in each part."""
    return torch.view_as_complex(torch.randn(*shape, 2, generator=g, device=DEV, dtype=torch.float64))


def _mul3(a, b):
    """3x3 products of two lists of nine whole-lattice arrays."""
    out = []
    for i in range(3):
        for j in range(3):
            t = a[3 * i] * b[j]
            t = torch.addcmul(t, a[3 * i + 1], b[3 + j])
            out.append(torch.addcmul(t, a[3 * i + 2], b[6 + j]))
    return out


def _links(L, eps, g):
    """exp(i eps H) with H traceless Hermitian from unit complex normals: [mu][3][3][T][Z][Y][X]."""
    shape = (L[3], L[2], L[1], L[0])
    U = torch.empty((4, 3, 3) + shape, dtype=C128, device=DEV)
    for mu in range(4):
        z = _normal((3, 3) + shape, g)
        h = 0.5 * (z + z.transpose(0, 1).conj())
        tr = (h[0, 0] + h[1, 1] + h[2, 2]) / 3.0
        x = [(1j * eps) * (h[i, j] - tr if i == j else h[i, j]) for i in range(3) for j in range(3)]
        del z, h
        one = [1.0 if i == j else 0.0 for i in range(3) for j in range(3)]
        p = [x[k] / 18.0 + one[k] for k in range(9)]
        for n in range(17, 0, -1):
            p = [v / n + o for v, o in zip(_mul3(x, p), one)]
        for k in range(9):
            U[mu, k // 3, k % 3] = p[k]
    return U


def _host_links(U):
    """Gauge::M layout [site][mu][3][3][re, im] in host memory."""
    m = U.permute(3, 4, 5, 6, 0, 1, 2).contiguous()
    return torch.view_as_real(m).reshape(-1, 4, 3, 3, 2).cpu().numpy()


class _Field:
    """A device spinor in the library's even-odd layout, held by torch."""

    def __init__(self, t):
        self.t = t
        self.ptr = t.data_ptr()


def _random_field(L, g):
    return _Field(_normal((2, 12, _volume(L) // 2), g))


def _empty_field(L):
    return _Field(torch.zeros((2, 12, _volume(L) // 2), dtype=C128, device=DEV))


def _sites(L):
    """Lexicographic index of every site of [parity][V/2]."""
    cb = torch.arange(_volume(L) // 2, device=DEV)
    j = 2 * cb
    r = torch.div(j, L[0], rounding_mode="floor")
    y = r % L[1]
    r = torch.div(r, L[1], rounding_mode="floor")
    s = y + r % L[2] + torch.div(r, L[2], rounding_mode="floor")
    return torch.stack([j + (s + p) % 2 for p in (0, 1)])


def _to_lex(f, L):
    """[2][12][V/2] -> [4][3][T][Z][Y][X]"""
    out = torch.empty((12, _volume(L)), dtype=C128, device=DEV)
    idx = _sites(L)
    for p in (0, 1):
        out[:, idx[p]] = f[p]
    return out.reshape(4, 3, L[3], L[2], L[1], L[0])


def _to_eo(f, L):
    f = f.reshape(12, -1)
    idx = _sites(L)
    return torch.stack([f[:, idx[p]] for p in (0, 1)])


def _eps(seed):
    return 0.2 + 0.1 * ((int(seed) * 7) % 11) / 10.0


def _point_sources(L, nrhs, seed):
    V = _volume(L)
    site = (int(seed) * 7919 + 13) % V
    x0, rest = site % L[0], site // L[0]
    y, z, t = rest % L[1], rest // L[1] % L[2], rest // L[1] // L[2]
    par = (x0 + y + z + t) % 2
    out = []
    for r in range(nrhs):
        f = _empty_field(L)
        f.t[par, r % 12, site // 2] = 1.0
        out.append(f)
    return out


def _lattice_for(case, L, U):
    lat = qkx.Lattice(qkx.LatticeInfo(L=L, kappa=KAPPA, mu=case.get("mu", 0.004), twistSign=1, boundaryT=-1))
    lat.load_gauge(_host_links(U), qkx.LINKS_APPLY_BC)
    return lat


def _sources(case, L, seed, salt):
    if case.get("source") == "point":
        return _point_sources(L, case["nrhs"], seed)
    g = _rng(seed, salt)
    return [_random_field(L, g) for _ in range(case["nrhs"])]


def _batch_lattices(case):
    """The three volumes of a batch: the case's lattice and two smaller ones."""
    L = _dims(case)

    def part(v, num, den):
        return max(4, 2 * (v * num // den // 2))

    return [L, tuple(part(v, 3, 4) for v in L), tuple(part(v, 1, 2) for v in L)]


def prepare(case, seed):
    L = _dims(case)
    kind = case["kind"]
    s = {"case": case}
    if kind == "blas":
        g = _rng(seed, 2)
        s["lat"] = qkx.Lattice(qkx.LatticeInfo(L=L))
        s["f"] = [_random_field(L, g) for _ in range(4)]
    elif kind == "twopt":
        s["lat"] = qkx.Lattice(qkx.LatticeInfo(L=L))
        s["p"] = _propagators(L, seed)
        s["src"] = tuple((int(seed) * 5 + 3 * i) % L[i] for i in range(4))
    elif kind == "batch":
        s["jobs"] = []
        for k, Lk in enumerate(_batch_lattices(case)):
            lat = _lattice_for(case, Lk, _links(Lk, _eps(seed + k), _rng(seed, 10 + k)))
            bs = _sources(case, Lk, seed, 20 + k)
            s["jobs"].append((lat, bs, [_empty_field(Lk) for _ in bs], [case["mu"]] * len(bs)))
    else:
        U = _links(L, _eps(seed), _rng(seed, 1))
        if kind == "smear":
            s["lat"] = qkx.Lattice(qkx.LatticeInfo(L=L))
            s["lat"].load_smearing_gauge(_host_links(U))
        else:
            s["lat"] = _lattice_for(case, L, U)
        if kind == "op":
            s["in"] = [_random_field(L, _rng(seed, 2))]
        else:
            s["in"] = _sources(case, L, seed, 2)
        s["out"] = [_empty_field(L) for _ in s["in"]]
    torch.cuda.synchronize()  # the inputs are ready before the library's own stream reads them
    return s


def _propagators(L, seed):
    """Two propagators [site][4][4][3][3] whose size falls off with the time distance, as a quark's does."""
    g = _rng(seed, 3)
    V3 = L[0] * L[1] * L[2]
    t = torch.arange(L[3], device=DEV, dtype=torch.float64)
    w = torch.exp(-0.1 * torch.minimum(t, L[3] - t)).reshape(-1, 1, 1)
    out = []
    for _ in range(2):
        p = _normal((L[3], V3, 144), g)
        p *= w
        out.append(p)
    return out


# ------------------------------------------------------------------ the pass
ALPHA, BETA = 0.0371, 0.613


def run(s):
    case, lat = s["case"], s.get("lat")
    kind = case["kind"]
    if kind == "op":
        lat.apply_dev(case["op"], s["in"][0], s["out"][0])
        return s["out"][0].t
    if kind == "blas":
        x, r, p, ap = s["f"]
        pap = lat.reCdotXdagY(p, ap)
        lat.X_eq_X_p_aY(x, ALPHA, p)
        lat.X_eq_X_p_aY(r, -ALPHA, ap)
        r2 = lat.norm2(r)
        lat.X_eq_aX_p_Y(p, BETA, r)
        return [pap, r2, x.t, r.t, p.t]
    if kind == "solve":
        method = qkx.SOLVER_CG_FP64 if case["method"] == "fp64" else qkx.SOLVER_CG_EO_MIXED
        lat.invert_dev(s["in"], s["out"], method=method, precision=PREC[case["precision"]], tol=case["tol"])
        return [f.t for f in s["out"]]
    if kind == "batch":
        qkx.invert_batch(s["jobs"], tol=case["tol"])
        return [f.t for job in s["jobs"] for f in job[2]]
    if kind == "smear":
        lat.Gaussian_smearing_dev(s["in"], s["out"], nsmear=case["nsmear"], alpha=4.0)
        return [f.t for f in s["out"]]
    p1, p2 = s["p"]
    return [lat.meson_2pt(p1.data_ptr(), Q_sq=case["qsq"], x_src=s["src"], device=True),
            lat.nucleon_2pt(p1.data_ptr(), p2.data_ptr(), Q_sq=case["qsq"], x_src=s["src"], device=True)]


# ------------------------------------------------------------------ the work
SPINOR, LINK = 192.0, 144.0  # FP64 bytes of a spinor and of a link
HOP_FLOPS = 1320.0           # of the hopping term, per site


def work(case):
    """Bytes and operations of one pass, inputs and outputs once each.  Iterative calls: the passes over memory
    that the method cannot do without -- a smearing step reads and writes every field (they exceed the caches),
    and a solve is counted as its right-hand sides in, solutions out and links in, with the hops of as many
    normal-operator applications as the plain (60) or even-odd (40) CG takes for the arithmetic."""
    L = _dims(case)
    V = _volume(L)
    kind = case["kind"]
    if kind == "op":
        op = case["op"]
        half = op.startswith("tm_xx")
        hops = 2 if op.startswith("tm_dagtm") else (2 if "dagtm" in op else 1)
        # in one parity and out the whole field (the reference's zero half is written) for the Schur operators
        io = (0.5 + 1.0 if half else 2.0) * SPINOR
        return {"bytes": V * (io + 4 * LINK), "flops": V * HOP_FLOPS * hops}
    if kind == "blas":
        return {"bytes": 12 * SPINOR * V, "flops": V * 24.0 * 10}
    if kind == "solve":
        n = case["nrhs"]
        its = 120.0 if case["method"] == "fp64" else 80.0
        return {"bytes": V * (2 * SPINOR * n + 4 * LINK), "flops": V * HOP_FLOPS * its * n}
    if kind == "batch":
        w = [work(dict(case, kind="solve", method="mixed", lx=l[0], ly=l[1], lz=l[2], lt=l[3]))
             for l in _batch_lattices(case)]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    if kind == "smear":
        n, k = case["nrhs"], case["nsmear"]
        return {"bytes": k * V * (2 * SPINOR * n + 3 * LINK), "flops": k * V * n * 6 * 264.0}
    return {"bytes": V * 2 * 2304.0, "flops": V * (10 * 16 * 9 * 8.0 + 3600 * 8.0)}


# ------------------------------------------------------------------ the same results in 64 bits
def _gammas(basis):
    """gamma_1..gamma_4, gamma_5 as (column, entry) of each row."""
    if basis == "ukqcd":
        return [[(3, 1j), (2, 1j), (1, -1j), (0, -1j)], [(3, 1), (2, -1), (1, -1), (0, 1)],
                [(2, 1j), (3, -1j), (0, -1j), (1, 1j)], [(0, 1), (1, 1), (2, -1), (3, -1)],
                [(2, 1), (3, 1), (0, 1), (1, 1)]]
    return [[(3, -1j), (2, -1j), (1, 1j), (0, 1j)], [(3, -1), (2, 1), (1, 1), (0, -1)],
            [(2, -1j), (3, 1j), (0, 1j), (1, -1j)], [(2, -1), (3, -1), (0, -1), (1, -1)],
            [(0, 1), (1, 1), (2, -1), (3, -1)]]


class _Wilson:
    """The hopping term and the operators on [4][3][T][Z][Y][X] fields, links [mu][3][3][T][Z][Y][X]."""

    def __init__(self, U, L, mu, basis="ukqcd"):
        self.U = U.clone()
        self.U[3, :, :, L[3] - 1] *= -1.0  # antiperiodic in time
        self.c = 2.0 * KAPPA * mu
        self.g = _gammas(basis)
        x = [torch.arange(n, device=DEV) for n in L]
        par = x[3].reshape(-1, 1, 1, 1) + x[2].reshape(-1, 1, 1) + x[1].reshape(-1, 1) + x[0]
        self.even = (par % 2 == 0).to(torch.float64)

    def gamma(self, m, psi):
        return torch.stack([e * psi[c] for c, e in self.g[m]])

    def dslash(self, psi, dag=False):
        out = torch.zeros_like(psi)
        sf = 1.0 if dag else -1.0
        for m in range(4):
            dim = -1 - m
            for fwd in (True, False):
                sign = sf if fwd else -sf
                v = psi + sign * self.gamma(m, psi)
                if fwd:
                    v = torch.roll(v, -1, dim)
                u = self.U[m]
                w = torch.empty_like(v)
                for a in range(3):
                    if fwd:
                        t = u[a, 0] * v[:, 0]
                        t = torch.addcmul(t, u[a, 1].expand_as(t), v[:, 1])
                        w[:, a] = torch.addcmul(t, u[a, 2].expand_as(t), v[:, 2])
                    else:
                        t = u[0, a].conj() * v[:, 0]
                        t = torch.addcmul(t, u[1, a].conj().expand_as(t), v[:, 1])
                        w[:, a] = torch.addcmul(t, u[2, a].conj().expand_as(t), v[:, 2])
                out += w if fwd else torch.roll(w, 1, dim)
        return out

    def twist(self, psi, c):
        return psi + (1j * c) * self.gamma(4, psi)

    def tm(self, psi, dag=False, c=None):
        c = self.c if c is None else c
        return self.twist(psi, -c if dag else c) - KAPPA * self.dslash(psi, dag)

    def schur(self, psi, even, c):
        """A psi - kappa^2 D A^-1 D psi on one parity."""
        keep = self.even if even else 1.0 - self.even
        t = self.dslash(psi * keep) * (1.0 - keep)
        t = self.twist(t, -c) / (1.0 + c * c)
        return (self.twist(psi, c) - KAPPA**2 * self.dslash(t)) * keep

    def apply(self, op, psi):
        if op.startswith("tm_xx"):
            even = op.endswith("ee")
            c = self.c
            if "dagtm" not in op:
                return self.schur(psi, even, c)
            return self.gamma(4, self.schur(self.gamma(4, self.schur(psi, even, c)), even, -c))
        if op in ("tm", "tm_chiral"):
            return self.tm(psi)
        if op == "tm_dag":
            return self.tm(psi, dag=True)
        if op == "tm_dagtm":
            return self.tm(self.tm(psi), dag=True)
        if op == "wilson":
            return self.tm(psi, c=0.0)
        return self.dslash(psi)

    def solve(self, b):
        """x with M x = b: CG on M^+ M, restarted from the true residual until that stops falling."""
        x = torch.zeros_like(b)
        bn = float(torch.linalg.vector_norm(b))
        best = math.inf
        for _ in range(6):
            res = b - self.tm(x)
            rel = float(torch.linalg.vector_norm(res)) / bn
            if rel < 1e-14 or rel > 0.5 * best:
                break
            best = rel
            r = self.tm(res, dag=True)
            p = r.clone()
            r2 = float(torch.linalg.vector_norm(r)) ** 2
            stop = r2 * 1e-22
            for _ in range(400):
                q = self.tm(p)
                a = r2 / float(torch.linalg.vector_norm(q)) ** 2
                x += a * p
                r -= a * self.tm(q, dag=True)
                new = float(torch.linalg.vector_norm(r)) ** 2
                p = r + (new / r2) * p
                r2 = new
                if r2 < stop:
                    break
        return x


def _exact_solve(case, L, U, sources, count):
    """Solutions of the first `count` sources, None for the others."""
    w = _Wilson(U, L, case["mu"])
    out = []
    for k, f in enumerate(sources):
        out.append(_to_eo(w.solve(_to_lex(f.t, L)), L) if k < count else None)
    return out


def _momenta(qsq):
    return [(x, y, z) for q in range(qsq + 1) for x in range(q, -q - 1, -1) for y in range(q, -q - 1, -1)
            for z in range(q, -q - 1, -1) if x * x + y * y + z * z == q]


def _fourier(c, L, qsq, src):
    """c [T][V3][K] -> [T][momentum][K], exp(-2 pi i p (x - x_src) / L) with the reference's value of pi."""
    pi = 3.14159265359
    x = torch.arange(L[0], device=DEV, dtype=torch.float64) - src[0]
    y = (torch.arange(L[1], device=DEV, dtype=torch.float64) - src[1]).reshape(-1, 1)
    z = (torch.arange(L[2], device=DEV, dtype=torch.float64) - src[2]).reshape(-1, 1, 1)
    ph = []
    for n in _momenta(qsq):
        th = (n[0] * x / L[0] + n[1] * y / L[1] + n[2] * z / L[2]) * 2 * pi
        ph.append(torch.polar(torch.ones_like(th), -th).reshape(-1))
    return torch.einsum("mv,tvk->tmk", torch.stack(ph), c)


def _dense(rows):
    m = torch.zeros((4, 4), dtype=C128, device=DEV)
    for r, (c, e) in enumerate(rows):
        m[r, c] = e
    return m


def _exact_twopt(case, L, seed):
    p1, p2 = (p.reshape(L[3], -1, 4, 4, 3, 3) for p in _propagators(L, seed))
    src = tuple((int(seed) * 5 + 3 * i) % L[i] for i in range(4))
    G = [_dense(r) for r in _gammas("ukqcd")]
    ops = [torch.eye(4, dtype=C128, device=DEV), G[4]] + G[:4] + [G[4] @ g for g in G[:4]]
    Cm = G[1] @ G[3]
    cg = Cm @ G[4]
    cgbar = G[3] @ cg.conj().T @ G[3]
    eps = torch.zeros((3, 3, 3), dtype=C128, device=DEV)
    for a, b, c, v in ((0, 1, 2, 1), (1, 2, 0, 1), (2, 0, 1, 1), (2, 1, 0, -1), (0, 2, 1, -1), (1, 0, 2, -1)):
        eps[a, b, c] = v
    mes, bar = [], []
    for t in range(L[3]):
        P, Q = p1[t], p2[t]
        back = torch.einsum("mk,vlkba,ln->vmnab", G[4], P.conj(), G[4])
        cols = []
        for g in ops:
            # tr[g (g5 P^+ g5) g P]
            cols.append(torch.einsum("vsgba,vgsab->v", torch.einsum("vgdba,ds->vgsba", back, g).transpose(1, 2),
                                     torch.einsum("vsbxy,bg->vsgxy", P, g).transpose(1, 2)))
        mes.append(torch.stack(cols, -1))
        W = torch.einsum("xy,vyzbc,zw->vxwbc", cg, Q, cgbar)  # [alpha][alpha']
        D = torch.einsum("abc,vxwbB->vxwacB", eps, W)
        K = torch.einsum("ABC,vxwacB->vxwacAC", eps, D)       # eps eps W over the second quark's colours
        S = torch.einsum("vxwacAC,vxwaA->vcC", K, P)
        b1 = torch.einsum("vcC,vghcC->vgh", S, P)
        R = torch.einsum("vxwacAC,vgwcA->vxgaC", K, P)
        b2 = torch.einsum("vxgaC,vxhaC->vgh", R, P)
        bar.append((b1 - b2).reshape(-1, 16))
    m = _fourier(torch.stack(mes), L, case["qsq"], src).permute(2, 0, 1)
    n = _fourier(torch.stack(bar), L, case["qsq"], src).reshape(L[3], -1, 4, 4)
    return [torch.view_as_real(v.contiguous()).cpu().numpy() for v in (m, n)]


def exact(case, seed):
    L = _dims(case)
    kind = case["kind"]
    if kind == "blas":
        g = _rng(seed, 2)
        x, r, p, ap = (_random_field(L, g).t for _ in range(4))
        pap = float(torch.sum(p.real * ap.real + p.imag * ap.imag))
        x = x + ALPHA * p
        r = r - ALPHA * ap
        r2 = float(torch.sum(r.real * r.real + r.imag * r.imag))
        return [pap, r2, x, r, BETA * p + r]
    if kind == "twopt":
        return _exact_twopt(case, L, seed)
    if kind == "batch":
        out = []
        for k, Lk in enumerate(_batch_lattices(case)):
            U = _links(Lk, _eps(seed + k), _rng(seed, 10 + k))
            out += _exact_solve(case, Lk, U, _sources(case, Lk, seed, 20 + k), 2)
        return out
    U = _links(L, _eps(seed), _rng(seed, 1))
    if kind == "op":
        basis = "chiral" if "chiral" in case["op"] else "ukqcd"
        psi = _to_lex(_random_field(L, _rng(seed, 2)).t, L)
        return _to_eo(_Wilson(U, L, case["mu"], basis).apply(case["op"], psi), L)
    if kind == "solve":
        return _exact_solve(case, L, U, _sources(case, L, seed, 2), 1 if _volume(L) > 10**6 else 3)
    # smearing: psi <- (psi + alpha sum of the six spatial transports) / (1 + 6 alpha)
    out = []
    for k, f in enumerate(_sources(case, L, seed, 2)):
        if k >= 3:
            out.append(None)
            continue
        psi = _to_lex(f.t, L)
        for _ in range(case["nsmear"]):
            acc = torch.zeros_like(psi)
            for m in range(3):
                v = torch.roll(psi, -1, -1 - m)
                acc += torch.stack([(U[m, a].unsqueeze(0) * v).sum(1) for a in range(3)], 1)
                w = torch.stack([(U[m, :, a].conj().unsqueeze(0) * psi).sum(1) for a in range(3)], 1)
                acc += torch.roll(w, 1, -1 - m)
            psi = (psi + 4.0 * acc) / (1.0 + 24.0)
        out.append(_to_eo(psi, L))
    return out
