"""The calls whose speed is measured, with their inputs and their values in 64 bits.

Each case is one call (or the short sequence) that a propagation program makes
through the package's public entry points on device-resident state.  Orbitals are
Gaussians of width 1 bohr times complex noise, orthonormalised; A-vectors are
normalised complex noise; nuclei sit on the grid or half-grid positions that the
sinc-DVR project asks for.
"""
import itertools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "v1-1_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from sincgpu import Batch, SincProject, WalkTables, inputs  # noqa: E402

DT = 0.05  # au, the time step of the propagation configurations


def _case(name, kind, points, spacing, nspf, elec, shift, charge1, charge2, **more):
    # nuclei of the two charges at z = +-shift half-grid steps (one nucleus at the
    # centre when charge2 is 0)
    return dict(name=name, kind=kind, points=points, spacing=spacing, nspf=nspf, elec=elec, shift=shift,
                charge1=charge1, charge2=charge2, **more)


def listed():
    return [
        # one orbital-RHS evaluation from the A-vector (mean fields, reduced potentials,
        # twoematel, RHS), what every step of a propagation is made of: the smallest
        # system (He, launch latency counts) ...
        _case("rhs 21^3 5 orbitals", "rhs", 21, 0.4, 5, 2, 0, 2.0, 0.0),
        # ... the H2-like system of the drop-in configuration ...
        _case("rhs 41^3 10 orbitals", "rhs", 41, 0.25, 10, 2, 6, 1.0, 1.0),
        # ... an odd electron and orbital count on a middle grid, as the mixed streams draw them ...
        _case("rhs 57^3 11 orbitals", "rhs", 57, 0.31, 11, 3, 4, 2.0, 1.0),
        # ... and the largest configuration (LiH-like, 14400 determinants, the benchmark's headline)
        _case("rhs 81^3 16 orbitals", "rhs", 81, 0.3, 16, 4, 10, 3.0, 1.0),
        # the same evaluation in the precision form (FP32 Coulomb passes, 3xTF32 reducedpot)
        _case("rhs mixed 81^3 16 orbitals", "rhs", 81, 0.3, 16, 4, 10, 3.0, 1.0, mixed=True),
        # the drop-in Coulomb call of a driver that builds its mean fields itself, with
        # different bra and ket orbitals, on an even grid
        _case("twoe 48^3 6 orbitals", "twoe", 48, 0.3, 6, 2, 5, 2.0, 1.0),
        # one orbital Krylov matvec as a driver's own exponential propagator calls it:
        # actreduced with the mean fields of the step, inside a pulse
        _case("matvec 41^3 10 orbitals", "matvec", 41, 0.25, 10, 2, 6, 1.0, 1.0),
        # one CI sigma product of the 14400-determinant space, with the field
        _case("sigma 14400 determinants", "sigma", 21, 0.4, 16, 4, 0, 4.0, 0.0),
        # the A-vector's Krylov propagation over one step in a middle CI space
        _case("avector step 3136 determinants", "avec", 21, 0.4, 8, 6, 0, 6.0, 0.0),
        # the orbitals' Krylov propagation over one mean-field interval
        _case("orbital step 41^3 10 orbitals", "spf", 41, 0.25, 10, 2, 6, 1.0, 1.0),
        # a served request's work: start and first step of a propagation in a pulse
        _case("cmf step 31^3 8 orbitals", "cmf", 31, 0.3, 8, 4, 4, 3.0, 1.0),
        # eight small systems of uneven size in one captured-graph launch
        dict(name="batch of 8", kind="batch", count=8, draw=2024, configs=1000),
    ]


_LARGEST = 81


def draw(rng):
    """One more case of the same ranges: grids of 21 to 81 points a side (even ones
    too), 4 to 16 orbitals, 2 to 6 electrons, up to 14400 determinants."""
    kind = rng.choice(["rhs", "rhs", "rhs", "mixed", "twoe", "matvec", "sigma", "avec", "spf", "cmf"])
    top = {"twoe": 57, "spf": 57, "cmf": 41, "sigma": 25, "avec": 25}.get(kind, _LARGEST)
    points = int(round(math.exp(rng.uniform(math.log(21), math.log(top)))))
    spacing = round(rng.uniform(0.25, 0.4), 3)
    elec = rng.randint(2, 6)
    most = {"avec": 4000, "cmf": 4000}.get(kind, 14400)
    nspf = rng.randint(max(4, (elec + 1) // 2 + 1), {"twoe": 9, "cmf": 9}.get(kind, 16))
    while nspf > (elec + 1) // 2 + 1 and inputs.ci_size(elec, nspf) > most:
        nspf -= 1
    two = rng.random() < 0.6
    shift = rng.randint(1, 5) * 2 - (points + 1) % 2 if two else 0
    c = _case("", "rhs" if kind == "mixed" else kind, points, spacing, nspf, elec, shift,
              float(rng.randint(1, 3)), float(rng.randint(1, 3)) if two else 0.0)
    if kind == "mixed":
        c["mixed"] = True
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _systems(case):
    """The systems of a case: grid, spacing, nuclei (half-grid steps), orbitals, electrons."""
    if case["kind"] == "batch":
        return inputs.batched_instances(case["count"], case["draw"], case["configs"])
    s, off = case["shift"], 1 - case["points"] % 2  # nuclei of an even grid sit half a step off its centre
    if case["charge2"]:
        shifts, charges = ((off, off, s), (off, off, -s)), (case["charge1"], case["charge2"])
    else:
        shifts, charges = ((off, off, off),), (case["charge1"],)
    return [dict(numpoints=case["points"], spacing=case["spacing"], centershift=shifts, nuccharges=charges,
                 nspf=case["nspf"], numelec=case["elec"], restrictms=case["elec"] % 2)]


def _noise(gen, *shape):
    return torch.complex(torch.randn(*shape, generator=gen, dtype=torch.float64, device="cuda"),
                         torch.randn(*shape, generator=gen, dtype=torch.float64, device="cuda"))


def _orbitals(gen, s):
    """nspf orthonormal orbitals, shape (nspf, N^3), x fastest."""
    N, n = s["numpoints"], s["nspf"]
    p = torch.arange(N, dtype=torch.float64, device="cuda")
    p = (p - (N - 1) / 2) * s["spacing"]
    r2 = p[:, None, None] ** 2 + p[None, :, None] ** 2 + p[None, None, :] ** 2
    phi = _noise(gen, n, N ** 3) * torch.exp(-r2 / 2).reshape(1, -1)
    low = torch.linalg.cholesky(phi.conj() @ phi.T)
    return torch.linalg.solve_triangular(low.conj(), phi, upper=False).contiguous()


def _avector(gen, s):
    a = _noise(gen, inputs.ci_size(s["numelec"], s["nspf"]))
    return a / torch.linalg.vector_norm(a)


def _project(s):
    p = SincProject(s["numpoints"], s["spacing"], s["centershift"], s["nuccharges"], s["nspf"])
    p.set_stream(torch.cuda.current_stream().cuda_stream)
    return p


def _buffers(s):
    n, G = s["nspf"], s["numpoints"] ** 3

    def z(*shape):
        return torch.zeros(*shape, dtype=torch.complex128, device="cuda")

    # Fortran arrays: the first index of the reference's arrays is the last one here
    return dict(denmat=z(n, n), invdenmat=z(n, n), tally=z(n, n, n, n), twoematel=z(n, n, n, n),
                reducedpot=z(n, n, G), out=z(n, G))


def _rhs(p, phi, avec, b, field=0.0):
    p.orbital_rhs_avec_dev(phi, avec, b["denmat"], b["invdenmat"], b["tally"], b["twoematel"], b["reducedpot"],
                           b["out"], ztdpot=field)


class _Pulse:  # one sin^2 pulse, as the served configuration draws them
    pulsetype, omega, omega2, pulsestart, phaseshift = 2, math.pi / 800, 0.3, 0.0, 0.0
    strength, longstep, pulsetheta = 0.05 / 0.3, 0.0, 0.0


def _inputs(case, seed):
    """What the seed alone makes: per system (system, orbitals, A-vector(s), field)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    out = []
    for s in _systems(case):
        kind = case["kind"]
        phi = _orbitals(gen, s)
        second = _orbitals(gen, s) if kind == "twoe" else None
        avecs = [_avector(gen, s) for _ in range(2 if kind == "spf" else 1)] if kind != "twoe" else []
        field = 0.02 + 0.05 * torch.rand(1, generator=gen, device="cuda").item()
        out.append((s, phi, second, avecs, field))
    return out


def prepare(case, seed):
    kind = case["kind"]
    parts = []
    for s, phi, second, avecs, field in _inputs(case, seed):
        p = _project(s)
        if case.get("mixed"):
            p.set_option("coulomb_fp32", 1)
            p.set_option("contract_tf32", 1)
        if kind != "twoe":
            walks = WalkTables(s["numelec"], s["nspf"], s["restrictms"])
            if kind == "cmf":
                walks.build_spin()
            p.ci_attach(walks)
        b = _buffers(s)
        part = dict(p=p, phi=phi, second=second, avecs=avecs, field=field, b=b)
        if kind == "twoe":
            part["red"] = torch.zeros_like(b["reducedpot"])
        elif kind == "matvec":  # the mean fields of the step
            _rhs(p, phi, avecs[0], b)
        elif kind == "spf":  # mean fields at both ends of the interval
            slots = []
            for a in avecs:
                _rhs(p, phi, a, b)
                slots.append((b["denmat"].clone(), b["invdenmat"].clone(), b["reducedpot"].clone()))
            part["slots"], part["moved"] = slots, torch.empty_like(phi)
        elif kind in ("sigma", "avec"):  # the CI matrices of the step
            n = s["nspf"]
            mats = torch.zeros(3, n, n, dtype=torch.complex128, device="cuda")
            p.twoe_matel_dev(phi, phi, b["twoematel"])
            p.onebody_matel_dev(phi, mats)
            p.assemble_sparsemats_dev(b["twoematel"], mats)
            part["sigma"] = torch.zeros_like(avecs[0])
            part["host"] = avecs[0].cpu().numpy()  # the Krylov entry takes host arrays
        elif kind == "cmf":
            part["final"] = torch.empty_like(phi), torch.empty_like(avecs[0])
        elif kind == "batch":
            p.rhs_graph_capture(phi, avecs[0], b["denmat"], b["invdenmat"], b["tally"], b["twoematel"],
                                b["reducedpot"], b["out"])
        parts.append(part)
    state = dict(kind=kind, parts=parts)
    if kind == "batch":
        state["batch"] = Batch([part["p"] for part in parts])
    return state


def run(state):
    kind, part = state["kind"], state["parts"][0]
    p, phi, b, avecs = part["p"], part["phi"], part["b"], part["avecs"]
    if kind == "rhs":
        _rhs(p, phi, avecs[0], b)
        return b
    if kind == "twoe":
        p.twoe_matel_dev(phi, part["second"], b["twoematel"], part["red"])
        return {"twoematel": b["twoematel"], "twoereduced": part["red"]}
    if kind == "matvec":
        p.actreduced_dev(phi, phi, b["denmat"], b["invdenmat"], b["reducedpot"], b["out"], ztdpot=part["field"])
        return b["out"]
    if kind == "sigma":
        p.sparseconfigmult_dev(avecs[0], part["sigma"], part["field"])
        return part["sigma"]
    if kind == "avec":
        return p.expoavecprop(part["host"], 1.0, krylovdim=30, tol=1e-9, anorm=DT, timefac=-1j * DT,
                              ezfield=part["field"])[0]
    if kind == "spf":
        part["moved"].copy_(phi)
        p.orbprop_setup(first_stepsize=DT)
        p.expospfprop_dev(part["moved"], part["slots"][0], part["slots"][1], 0.0, DT, 0.0, DT, ezfield=part["field"])
        return part["moved"]
    if kind == "cmf":
        p.cmf_setup(par_timestep=DT)
        p.cmf_pulses([_Pulse])
        energy0 = p.cmf_init_dev(phi, avecs[0])
        step = p.cmf_step(0.0, DT)
        p.cmf_state_dev(*part["final"])
        return [energy0, step["energy"], step["norm"], *part["final"]]
    state["batch"].launch(torch.cuda.current_stream().cuda_stream)
    return [{k: q["b"][k] for k in ("denmat", "invdenmat", "tally", "twoematel", "reducedpot", "out")}
            for q in state["parts"]]


# ---------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------
def _coulomb_flops(N, solves):
    # per solve: 3-D transform of an N^3 density on the doubled grid and back, on
    # lines that are not zero (5 L log2 L each), and one real factor per frequency
    L = 2 * N
    return solves * (2 * (N * N + N * L + L * L) * 5 * L * math.log2(L) + 2 * L ** 3 + 6 * N ** 3)


def _kinetic_flops(N, n):
    return 3 * 4 * n * N ** 4


def _mean_field(N, n):
    G, pairs = N ** 3, n * (n + 1) / 2
    # hermitian pairs: n^2 real potentials; twoematel is symmetric
    return _coulomb_flops(N, pairs - n / 2) + G * n ** 4 + 2 * G * n ** 4


def _ci(s):
    """Determinants and (single, double) excitations per determinant."""
    n, ne = s["nspf"], s["numelec"]
    na = (ne + ne % 2) // 2
    nb = ne - na

    def singles(k):
        return k * (n - k)

    def doubles(k):
        return math.comb(k, 2) * math.comb(n - k, 2)

    one = 1 + singles(na) + singles(nb)
    return inputs.ci_size(ne, n), one, one + doubles(na) + doubles(nb) + singles(na) * singles(nb)


def work(case):
    kind = case["kind"]
    z = 16  # bytes of a complex number
    bytes_, flops = 0.0, 0.0
    for s in _systems(case):
        N, n = s["numpoints"], s["nspf"]
        G = N ** 3
        nc, one, two = _ci(s)
        matvec = _kinetic_flops(N, n) + 8 * G * n * n + 16 * G * n * n + 16 * G * n * n
        build = _mean_field(N, n) + 8.0 * nc * (one + two)
        if kind in ("rhs", "batch"):
            bytes_ += z * (2 * G * n + nc + 2 * n ** 4 + G * n * n)
            flops += build + matvec
        elif kind == "twoe":
            bytes_ += z * (2 * G * n + n ** 4 + G * n * n)
            flops += _coulomb_flops(N, n * n) + 8.0 * G * n ** 4
        elif kind == "matvec":
            bytes_ += z * (2 * G * n + G * n * n)
            flops += matvec
        elif kind == "sigma":
            bytes_ += z * 2 * nc + (z + 4) * nc * (one + two)
            flops += 8.0 * nc * (one + two)
        elif kind == "avec":  # thirty products in the Krylov space
            bytes_ += 30 * (z * 2 * nc + (z + 4) * nc * (one + two))
            flops += 30 * (8.0 * nc * (one + two) + 8.0 * 30 * nc)
        elif kind == "spf":  # some forty products
            bytes_ += 40 * z * (2 * G * n + G * n * n)
            flops += 40 * matvec
        elif kind == "cmf":  # three mean-field builds, some sixty products
            bytes_ += 60 * z * (2 * G * n + G * n * n)
            flops += 4 * build + 60 * matvec
    return {"bytes": int(bytes_), "flops": int(flops)}


# ---------------------------------------------------------------------------
# the same values in plain torch and numpy, in 64 bits
# ---------------------------------------------------------------------------
def _greens(N, spacing, nbig=240, nsmall=40):
    """Inverse of the sinc-DVR kinetic operator on the lattice, divided by spacing^3:
    values at differences -(N-1)..N-1 per axis (1/r far away, corrected near the origin
    so that it inverts the operator there)."""
    nbig = max(nbig, N - 1)
    dev = "cuda"
    f64 = dict(dtype=torch.float64, device=dev)
    big, sm = torch.arange(-nbig, nbig + 1, **f64), torch.arange(-nsmall, nsmall + 1, **f64)

    def inv_r(a, b, c):
        r = torch.sqrt(a[:, None, None] ** 2 + b[None, :, None] ** 2 + c[None, None, :] ** 2) * spacing
        return torch.where(r == 0, torch.zeros_like(r), spacing ** 3 / torch.where(r == 0, torch.ones_like(r), r))

    def kinetic(d):
        near = torch.where(d == 0, torch.ones_like(d), d)
        t = torch.where(d % 2 == 0, 1.0, -1.0) / (spacing * near) ** 2
        return torch.where(d == 0, torch.full_like(d, math.pi ** 2 / 6 / spacing ** 2), t)

    A = kinetic(big[None, :] - sm[:, None])
    t = inv_r(big, sm, sm)
    t = torch.einsum("ip,pjk->ijk", A, t)
    rest = -(t + t.permute(1, 0, 2) + t.permute(1, 2, 0))
    rest[nsmall, nsmall, nsmall] += 2 * math.pi
    e, w = torch.linalg.eigh(kinetic(sm[:, None] - sm[None, :]))

    def rotate(m, q):  # m on each of the three axes
        for _ in range(3):
            q = torch.tensordot(q, m, dims=([0], [1]))
        return q

    q = rotate(w.T, rest) / (e[:, None, None] + e[None, :, None] + e[None, None, :])
    q = rotate(w, q)
    out = torch.arange(-(N - 1), N, **f64)
    g = inv_r(out, out, out)
    m = min(nsmall, N - 1)
    o, c = slice(N - 1 - m, N + m), slice(nsmall - m, nsmall + m + 1)
    g[o, o, o] += q[c, c, c]
    return g / spacing ** 3


class _Plain:
    """Operators of one system, orbitals as (n, N, N, N) with axes (orbital, z, y, x)."""

    def __init__(self, s):
        self.s, self.N, self.n = s, s["numpoints"], s["nspf"]
        N = self.N
        self.green = _greens(N, s["spacing"])
        L = 2 * N
        k = torch.zeros(L, L, L, dtype=torch.float64, device="cuda")
        at = torch.arange(-(N - 1), N, device="cuda") % L
        k[at[:, None, None], at[None, :, None], at[None, None, :]] = self.green
        self.spectrum = torch.fft.fftn(k).real.contiguous()
        d = torch.arange(N, dtype=torch.float64, device="cuda")
        d = d[:, None] - d[None, :]
        near = torch.where(d == 0, torch.ones_like(d), d)
        kin = torch.where(d == 0, torch.full_like(d, math.pi ** 2 / 3),
                          2.0 * torch.where(d % 2 == 0, 1.0, -1.0) / near ** 2) / (2 * s["spacing"] ** 2)
        self.kin = kin.to(torch.complex128)
        self.points = (torch.arange(N, dtype=torch.float64, device="cuda") - (N - 1) / 2) * s["spacing"]
        pot = torch.zeros(N, N, N, dtype=torch.float64, device="cuda")
        for shift, charge in zip(s["centershift"], s["nuccharges"]):
            at = [torch.arange(N, device="cuda") + (-N + c + 1) // 2 + N - 1 for c in shift]
            pot -= charge * self.green[at[2][:, None, None], at[1][None, :, None], at[0][None, None, :]]
        self.pot = pot

    def coulomb(self, rho):
        N, L = self.N, 2 * self.N
        f = torch.fft.fftn(rho, s=(L, L, L), dim=(-3, -2, -1)) * self.spectrum
        return torch.fft.ifftn(f, dim=(-3, -2, -1))[..., :N, :N, :N]

    def grid(self, phi):
        return phi.reshape(-1, self.N, self.N, self.N)

    def twoe(self, bra, ket):
        """(twoematel[b2, a2, b1, a1], twoereduced[b, a, G]) of rho_ab = bra_a conj(ket_b)."""
        n, G = self.n, self.N ** 3
        one, two = self.grid(bra), self.grid(ket)
        red = torch.empty(n, n, G, dtype=torch.complex128, device="cuda")
        den = torch.empty_like(red)
        for b in range(n):
            for a in range(n):
                rho = one[a] * two[b].conj()
                den[b, a] = rho.reshape(-1)
                red[b, a] = self.coulomb(rho).reshape(-1)
        mat = red.reshape(n * n, G) @ den.reshape(n * n, G).T
        return mat.reshape(n, n, n, n), red

    def kinetic(self, f):
        out = torch.einsum("nzyx,xw->nzyw", f, self.kin)
        out += torch.einsum("nzyx,yw->nzwx", f, self.kin)
        out += torch.einsum("nzyx,zw->nwyx", f, self.kin)
        return out

    def act(self, phi, den, inv, reducedpot, field):
        """(1 - P) (-i) [(T + V + E z) (phi den) + W phi] inv, matrices as den[j, i] = (i, j)."""
        n, G = self.n, self.N ** 3
        f = self.grid(den @ phi.reshape(n, G))
        h = self.kinetic(f) + (self.pot + field * self.points[:, None, None]) * f
        h = h.reshape(n, G) + torch.einsum("ikg,kg->ig", reducedpot, phi)
        h = -1j * (inv @ h)
        return h - (h @ phi.conj().T) @ phi

    def onebody(self, phi):
        """<phi_i|op|phi_j> as [i, j] of the potential, the kinetic energy and z."""
        f = self.grid(phi)
        z = self.points[:, None, None].expand(self.N, self.N, self.N)
        return [phi.conj() @ g.reshape(self.n, -1).T for g in (self.pot * f, self.kinetic(f), z * f)]


class _PlainCI:
    """Full CI of the system in products of alpha and beta strings."""

    def __init__(self, s):
        n, ne = s["nspf"], s["numelec"]
        nup = (ne + s["restrictms"]) // 2
        ndn = ne - nup
        self.n = n
        up = list(itertools.combinations(range(n), nup))
        dn = list(itertools.combinations(range(n), ndn))
        self.shape = (len(dn), len(up))
        self.down, self.up = self._moves(dn), self._moves(up)
        # the determinant list: by the sorted spatial orbitals, then by the spins
        # (the reference's spin 1 is the one of negative m)
        dets = []
        for i, d in enumerate(dn):
            for j, u in enumerate(up):
                so = sorted([(o, 1) for o in d] + [(o, 2) for o in u])
                swaps = sum(1 for a, b in itertools.combinations([x[1] for x in so], 2) if a > b)
                dets.append((tuple(x[0] for x in so), tuple(x[1] for x in so), i * len(up) + j, -1.0 if swaps % 2 else 1.0))
        dets.sort()
        self.at = torch.tensor([d[2] for d in dets], device="cuda")
        self.sign = torch.tensor([d[3] for d in dets], dtype=torch.float64, device="cuda")

    def _moves(self, strings):
        """M[p, q] = a+_p a_q among the strings."""
        index = {s: i for i, s in enumerate(strings)}
        m = np.zeros((self.n, self.n, len(strings), len(strings)))
        for s in strings:
            for pos, q in enumerate(s):
                for p in range(self.n):
                    rest = s[:pos] + s[pos + 1:]
                    if p in rest:
                        continue
                    new = tuple(sorted(rest + (p,)))
                    m[p, q, index[new], index[s]] = (-1.0) ** (pos + new.index(p))
        return torch.from_numpy(m).to("cuda", torch.complex128)

    def to_strings(self, a):
        c = torch.zeros(self.shape[0] * self.shape[1], dtype=torch.complex128, device="cuda")
        c[self.at] = a * self.sign
        return c.reshape(self.shape)

    def to_list(self, c):
        return c.reshape(-1)[self.at] * self.sign

    def excite(self, c):
        """E_pq c for all p, q: [p, q, down, up]."""
        return torch.einsum("pqij,jk->pqik", self.down, c) + torch.einsum("pqij,kj->pqki", self.up, c)

    def densities(self, a):
        """denmat and tally in the memory order of the Fortran arrays (reversed indices)."""
        n, c = self.n, self.to_strings(a)
        e = self.excite(c).reshape(n, n, -1)
        one = torch.einsum("x,pqx->pq", c.reshape(-1).conj(), e)      # <E_pq>
        two = torch.einsum("cdx,bax->cdba", e.conj(), e)               # <E_dc E_ba>
        # tally(a,b,c,d) = <E_dc E_ba> - delta_bc <E_da>, stored as [d, c, b, a]
        tally = two.permute(1, 0, 2, 3).clone()
        tally -= torch.einsum("cb,da->dcba", torch.eye(n, dtype=torch.complex128, device="cuda"), one)
        return one, tally  # denmat(i, j) = <E_ji>: stored [j, i]

    def sigma(self, a, h, v, constant):
        """constant a + sum h[p, q] E_pq a + half the sum of v[d, c, b, a] (E_dc E_ba - delta_bc E_da) a."""
        n, c = self.n, self.to_strings(a)
        e = self.excite(c).reshape(n * n, -1)
        h = h - 0.5 * torch.einsum("dxxa->da", v)
        # sum over b, a of v[d, c, b, a] E_ba c, then E_dc of each
        w = (0.5 * v.reshape(n * n, n * n) @ e).reshape(n, n, *self.shape)
        out = torch.einsum("pqij,pqjk->ik", self.down, w) + torch.einsum("pqij,pqkj->ki", self.up, w)
        out = out + (h.reshape(1, -1) @ e).reshape(self.shape) + constant * c
        return self.to_list(out)


def _inverse(den):
    u, sv, vh = torch.linalg.svd(den)
    inv = torch.where(sv < 1e-10, torch.full_like(sv, 1e10), 1.0 / sv)
    return (vh.conj().T * inv) @ u.conj().T


def exact(case, seed):
    kind = case["kind"]
    if kind in ("avec", "spf", "cmf"):  # adaptive propagations: no closed value to their tolerance
        return None
    outs = []
    for s, phi, second, avecs, field in _inputs(case, seed):
        plain = _Plain(s)
        if kind == "twoe":
            mat, red = plain.twoe(phi, second)
            return {"twoematel": mat, "twoereduced": red}
        ci = _PlainCI(s)
        mat, red = plain.twoe(phi, phi)
        n = s["nspf"]
        if kind == "sigma":
            pot, kin, z = plain.onebody(phi)
            charges, shifts = s["nuccharges"], s["centershift"]
            repulsion = sum(charges[i] * charges[j] / (0.5 * s["spacing"] * math.dist(shifts[i], shifts[j]))
                            for i in range(len(charges)) for j in range(i))
            nuclear = _nuclear_dipole(s)
            return ci.sigma(avecs[0], pot + kin + field * z, mat, repulsion + field * nuclear)
        den, tally = ci.densities(avecs[0])
        inv = _inverse(den)
        # reducedpot(x, k, i) = sum_cd R_cd(x) tally(c, d, k, i)
        reducedpot = (tally.reshape(n * n, n * n) @ red.reshape(n * n, -1)).reshape(n, n, -1)
        del red
        out = plain.act(phi, den, inv, reducedpot, field if kind == "matvec" else 0.0)
        if kind == "matvec":
            return out
        outs.append(dict(denmat=den, invdenmat=inv, tally=tally, twoematel=mat, reducedpot=reducedpot, out=out))
    return outs[0] if kind == "rhs" else outs


def _nuclear_dipole(s):
    return sum(c * 0.5 * s["spacing"] * shift[2] for shift, c in zip(s["centershift"], s["nuccharges"]))
