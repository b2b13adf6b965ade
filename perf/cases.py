"""Performance cases of the walker engine: what its users run, over the sizes they run it at.

The framework's work is the walker loop of a quantum Monte Carlo run, reached through
``mainline_b200.engine.Engine``: VMC and DMC blocks on a resident population, and, for programs
that keep the loop to themselves, the full evaluation of a set of walkers, single-electron move
ratios and orbital rows at given positions.  Systems are the seeded decks of
``mainline_b200.systems``: the two-atom molecule (all-electron and with pseudopotentials),
molecules of 4 to about 100 electrons, and periodic cells of the 8-atom, 32-electron family, at
the Gamma point or a k-point.

Mixed-precision contexts compute in FP32, so what they return is handed on in FP32 here, the
accuracy it has; FP64 contexts return FP64.
"""
from __future__ import annotations

import atexit
import itertools
import math
import re
import shutil
import tempfile

import numpy as np

from mainline_b200 import engine, systems

PRECISION = {"fp64": engine.FP64, "mixed": engine.MIXED}
VMC_TAU = 0.3


def listed():
    return [
        # a program that makes its own moves asks for one trial move of each of a few walkers: latency
        dict(name="ratio 64 walkers", call="ratio", system="n2_pseudo", electrons=14, precision="fp64", walkers=64),
        # local energies of one small set of all-electron walkers (an optimiser's or a checker's sample)
        dict(name="evaluate all-electron", call="evaluate", system="n2_allelectron", electrons=14, precision="fp64",
             walkers=256),
        # the same for a medium molecule in mixed precision, an odd electron count and a ragged population
        dict(name="evaluate molecule", call="evaluate", system="molecule", electrons=43, precision="mixed",
             walkers=1000),
        # orbitals, gradients and Laplacians of a periodic cell on a list of points (plots, densities, fits)
        dict(name="orbital rows cell", call="orbitals", system="cell", electrons=128, precision="mixed", walkers=1200),
        # VMC of the all-electron molecule with the small population of an equilibration or an optimisation step
        dict(name="vmc all-electron", call="vmc", system="n2_allelectron", electrons=14, precision="fp64",
             walkers=256, steps=20),
        # the headline: mixed-precision DMC of the pseudopotential molecule
        dict(name="dmc molecule", call="dmc", system="n2_pseudo", electrons=14, precision="mixed", walkers=4096,
             steps=10, tau=0.01),
        # the same physics in FP64 on a population that is no multiple of anything
        dict(name="dmc molecule fp64", call="dmc", system="n2_pseudo", electrons=14, precision="fp64", walkers=3001,
             steps=10, tau=0.01),
        # a few electrons and a very large population: launches, branching and copies weigh most
        dict(name="dmc large population", call="dmc", system="molecule", electrons=4, precision="mixed",
             walkers=65536, steps=10, tau=0.01),
        # a large molecule: determinants and orbitals that no longer fit in shared memory
        dict(name="dmc large molecule", call="dmc", system="molecule", electrons=72, precision="mixed", walkers=2048,
             steps=5, tau=0.01),
        # a solid in FP64: Ewald sums, image sums, three-body Jastrow
        dict(name="dmc cell fp64", call="dmc", system="cell", electrons=32, precision="fp64", walkers=1024, steps=5,
             tau=0.005),
        # the same solid with twisted boundary conditions and complex orbitals
        dict(name="dmc cell at a k-point", call="dmc", system="kcell", electrons=32, precision="mixed", walkers=2048,
             steps=5, tau=0.005),
        # the largest: a supercell of 32 atoms
        dict(name="dmc supercell", call="dmc", system="cell", electrons=128, precision="mixed", walkers=1024, steps=4,
             tau=0.005),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(["ratio", "evaluate", "orbitals", "vmc", "dmc", "dmc", "dmc"])
    precision = rng.choice(["fp64", "mixed"])
    system = rng.choice(["n2_allelectron", "n2_pseudo", "molecule", "molecule", "cell"] if call != "dmc" else
                        ["n2_pseudo", "molecule", "molecule", "cell", "kcell"])
    electrons = {"molecule": size(4, 96), "cell": 32, "kcell": 32}.get(system, 14)
    if system == "cell" and call in ("ratio", "orbitals") and rng.random() < 0.5:
        electrons = 128
    c = dict(call=call, system=system, electrons=electrons, precision=precision)
    if call in ("vmc", "dmc"):
        c["steps"] = rng.randint(2, 20) if call == "vmc" else rng.randint(2, 10)
    # at most about as many walker-steps as a quarter of the largest case's time allows
    heavy = 100.0 if system in ("cell", "kcell") else 20.0
    most = 5e8 / (heavy * electrons ** 2) / (c.get("steps", 1) + 1)
    c["walkers"] = size(64, max(128.0, min(65536.0, most)))
    if call == "dmc":
        c["tau"] = 0.005 if system in ("cell", "kcell") else 0.01
    return c


# ---- systems, walkers and contexts that a user's program has in hand

_folder = None
_decks = {}


def _deck(case):
    """The case's input deck, written once per process."""
    global _folder
    if _folder is None:
        _folder = tempfile.mkdtemp(prefix="qwg_cases_")
        atexit.register(shutil.rmtree, _folder, ignore_errors=True)
    key = (case["system"], case["electrons"])
    if key not in _decks:
        kind, n = key
        name = f"{kind}{n}"
        if kind.startswith("n2"):
            d = systems.write_n2(_folder, seed=12, pseudo=kind == "n2_pseudo", name=name)
        elif kind == "molecule":
            d = systems.write_molecule(_folder, name, seed=1000 + n, nelec=n)
        else:
            twist = dict(kpoint=(0.5, 0.25, 0.0), complex_orbitals=True) if kind == "kcell" else {}
            d = systems.write_periodic(_folder, seed=13, name=name, supercell={32: (1, 1, 1), 128: (2, 2, 1)}[n], **twist)
        _decks[key] = d
    return _decks[key]


def _walkers(case, seed):
    """Walkers as a run has them: started near the atoms and equilibrated by VMC (in FP64 whatever the case's precision)."""
    deck = _deck(case)
    e = engine.Engine(deck.path, engine.FP64, max_walkers=case["walkers"])
    e.set_walkers(systems.random_configs(deck, case["walkers"], seed=seed))
    e.vmc_block(3 if "cell" in case["system"] else 10, VMC_TAU, seed=seed + 1)
    r = e.get_walkers()
    e.close()
    return r


def prepare(case, seed):
    deck, rng = _deck(case), np.random.default_rng(seed)
    call, n = case["call"], case["walkers"]
    s = {"call": call, "fp32": case["precision"] == "mixed", "steps": case.get("steps"), "seed": seed}
    if call == "orbitals":  # positions of electrons, one each
        s["spin"] = seed % 2
        s["R"] = systems.random_configs(deck, n, seed=seed)[:, 0].copy()
        s["engine"] = engine.Engine(deck.path, PRECISION[case["precision"]], max_walkers=1)
        return s
    s["R"] = _walkers(case, seed)
    s["engine"] = engine.Engine(deck.path, PRECISION[case["precision"]], max_walkers=n)
    s["engine"].set_walkers(s["R"])
    if call == "ratio":
        s["electron"] = rng.integers(0, deck.nelec, size=n).astype(np.int32)
        s["to"] = s["R"][np.arange(n), s["electron"]] + rng.normal(0.0, 0.3, size=(n, 3))
    elif call == "evaluate":
        s["rot"] = np.stack([systems.random_rotation(rng) for _ in range(n)])
    elif call == "dmc":
        s["engine"].dmc_init(case["tau"], nstep=case["steps"], seed=seed + 2)
    return s


def run(state):
    e, call = state["engine"], state["call"]
    if call == "ratio":
        out = dict(zip(("dlogpsi", "sign", "grad", "lap"), e.ratio(state["electron"], state["to"])))
    elif call == "evaluate":
        r = e.eval(state["rot"])
        out = dict(logpsi=r.logpsi, sign=r.sign, grad=r.grad, lap=r.lap, kinetic=r.kinetic, potential=r.potential,
                   nonlocal_=r.nonlocal_)
    elif call == "orbitals":
        out = dict(rows=e.mo_eval(state["R"], state["spin"]))
    else:
        st = e.vmc_block(state["steps"], VMC_TAU, seed=state["seed"] + 3) if call == "vmc" else e.dmc_block()
        energy, weight = e.walker_scalars()
        out = {k: np.float64(v) if isinstance(v, float) else v for k, v in st.items() if k != "block_ms"}
        out.update(walkers=e.get_walkers(), walker_energy=energy, walker_weight=weight)
    if state["fp32"]:
        out = {k: v.astype(np.float32) if hasattr(v, "astype") else v for k, v in out.items()}
    return out


def _images(case):
    """Basis centers a position's image sums reach (the decks' 16 bohr cutoff), per atom of the cell."""
    if "cell" not in case["system"]:
        return 1.0
    return 4.0 / 3.0 * math.pi * 16.0 ** 3 / 6.74 ** 3 * 32.0 / case["electrons"]


def work(case):
    deck = _deck(case)
    n, nb, w = deck.nelec, deck.nbasis, case["walkers"]
    m, cplx = (n + 1) // 2, 4 if case["system"] == "kcell" else 1
    real = 4 if case["precision"] == "mixed" else 8
    table = 2 * nb * m * real
    row = 5 * (nb * 4 * _images(case) + nb * m * 2 * cplx)  # one position: basis functions and orbitals, five components
    pairs = 12 * ((n - 1) * 2 + deck.natoms * 4)            # one electron's Jastrow
    quad = 12 * 1.4 * n * (nb * 4 * _images(case) + 2 * nb + pairs) if case["system"] != "n2_allelectron" else 0
    sweep = n * (row + 10 * m + 4 * m * m + 5 * pairs)
    energy = n * (8 * m + 5 * n) + quad
    state = 8 * 3 * n
    if case["call"] == "orbitals":
        return dict(bytes=w * (24 + 40 * m) + table, flops=w * row)
    if case["call"] == "ratio":
        return dict(bytes=w * (28 + 48 + state) + table, flops=w * (row * (n + 1) + 2 * m ** 3))
    if case["call"] == "evaluate":
        return dict(bytes=w * (72 + state + 8 * (5 + 4 * n)) + table, flops=w * (n * row + 4 / 3 * m ** 3 + energy))
    return dict(bytes=w * (2 * state + 16) + table, flops=w * case["steps"] * (sweep + energy))


# ---- the same values in plain numpy, 64 bits, from the deck files

class _Plain:
    """A molecule's (or, for orbitals, a cell's) trial function as its deck states it."""

    def __init__(self, deck):
        text = open(deck.path).read()
        num = r"[-+0-9.eE]+"

        def floats(s):
            return [float(x) for x in s.split()]

        self.nup, self.n = deck.nup, deck.nelec
        atoms = re.findall(rf"ATOM \{{ (\S+) ({num}) COOR ({num}) ({num}) ({num}) \}}", text)
        self.label, self.z = [a[0] for a in atoms], np.array([float(a[1]) for a in atoms])
        self.at = np.array([[float(x) for x in a[2:]] for a in atoms])
        lat = re.search(r"LATTICEVEC \{([^}]*)\}", text)
        self.edge = np.array(floats(lat.group(1)))[[0, 4, 8]] if lat else None
        # radial splines on the 0.02 grid: contracted Gaussians with the GAMESS normalisation, renormalised
        # numerically, an optional smooth cutoff, a clamped cubic spline
        self.shells = {}
        for lab, head, body in re.findall(r"BASIS \{ (\S+)\s+AOSPLINE([^{}]*)GAMESS \{([^{}]*)\}", text):
            cut = re.search(rf"CUTOFF ({num})", head)
            self.shells[lab] = self._shells(body.split(), float(cut.group(1)) if cut else None)
        orb = open(deck.orb_path).read().split("COEFFICIENTS")
        coef = np.array(orb[1].split(), dtype=float)
        nmo = int(re.search(r"NMO (\d+)", text).group(1))
        self.mo = coef.reshape(nmo, -1).T
        st = [int(x) - 1 for x in re.search(r"STATES \{([^}]*)\}", text).group(1).split()]
        self.occ = [st[:self.nup], st[self.nup:]]
        # Jastrow: the cusp functions and the one-body polynomial Pade functions
        cusp = re.search(rf"CUTOFF_CUSP GAMMA ({num}) CUSP ({num}) CUTOFF ({num})", text)
        self.gamma, self.cusp, self.rcut = (float(x) for x in cusp.groups())
        self.ei = {lab: (float(b), int(k), float(rc)) for lab, b, k, rc in
                   re.findall(rf"EIBASIS \{{ (\S+) POLYPADE BETA0 ({num}) NFUNC (\d+) RCUT ({num})", text)}
        one = re.search(r"ONEBODY \{(.*?)\n  \}", text, re.S).group(1)
        self.one = {lab: floats(c) for lab, c in re.findall(r"COEFFICIENTS \{ (\S+) ([^}]*)\}", one)}
        self.pp = {}
        for lab, body in re.findall(r"PSEUDO \{ (\S+)\s+AIP 12\s+BASIS \{ \S+\s+RGAUSSIAN\s+OLDQMC \{([^}]*)\}", text):
            v = floats(body)
            count, v = [int(x) for x in v[2:5]], np.array(v[5:]).reshape(-1, 3)
            first = np.concatenate([[0], np.cumsum(count)])
            self.pp[lab] = [v[first[k]:first[k + 1]] for k in range(3)]

    @staticmethod
    def _shells(w, cut):
        h, n = 0.02, 2500
        x, out, p = np.arange(n) * h, [], 0
        while p < len(w):
            sym, k = w[p], int(w[p + 1])
            prim = np.array(w[p + 2:p + 2 + 3 * k], dtype=float).reshape(k, 3)
            p += 2 + 3 * k
            L = {"S": 0, "P": 1, "6D": 2}[sym]
            y = np.zeros(n)
            for _, a, c in prim:
                y += c * math.sqrt(2 * (4 * a) ** (L + 1) * math.sqrt(2 * a / math.pi) / (1, 3, 15)[L]) * np.exp(-a * x * x)
            s = np.sum(h * x ** (2 * L + 2) * y * y)
            if abs(s - 1) > 1e-5:
                y /= math.sqrt(s)
            if cut:
                z = (x - (cut - 1e-6 - 1.2)) / 1.2
                y = np.where(z > 1, 0, np.where(z > 0, y * (1 - z ** 3 * (6 * z * z - 15 * z + 10)), y))
            # second derivatives of the spline clamped to the end slopes of the table
            d, rhs = np.full(n, 4.0), np.zeros(n)
            dy = np.diff(y)
            rhs[1:-1] = 6 / h ** 2 * (dy[1:] - dy[:-1])
            d[0] = d[-1] = 2.0
            cp, dp = np.zeros(n), np.zeros(n)
            for i in range(n):
                low = 1.0 if i else 0.0
                m = d[i] - low * (cp[i - 1] if i else 0.0)
                cp[i], dp[i] = 1.0 / m, (rhs[i] - low * (dp[i - 1] if i else 0.0)) / m
            y2 = dp
            for i in range(n - 2, -1, -1):
                y2[i] -= cp[i] * y2[i + 1]
            c = np.zeros((n, 4))
            c[:-1] = np.stack([y[:-1], dy / h - h * (2 * y2[:-1] + y2[1:]) / 6, y2[:-1] / 2, np.diff(y2) / (6 * h)], 1)
            out.append((L, c))
        return out

    def basis(self, p, values_only=False):
        """Basis functions at positions p [n, 3]: [n, functions, 5] (or 1)."""
        q, out = 1 if values_only else 5, []
        for a, lab in enumerate(self.label):
            images = [np.zeros(3)]
            if self.edge is not None:
                reach = [range(-math.ceil(16 / e) - 1, math.ceil(16 / e) + 2) for e in self.edge]
                images = [np.array(t) * self.edge for t in itertools.product(*reach)]
            total = 0.0
            for t in images:
                f = np.zeros((len(p), sum((1, 3, 6)[L] for L, _ in self.shells[lab]), q))
                d = p - self.at[a] - t
                r = np.sqrt((d * d).sum(1))
                near = np.flatnonzero(r < (16.0 if self.edge is not None else 49.9))
                if len(near):
                    f[near] = self._center(d[near], r[near], self.shells[lab], values_only)
                    total = total + f
            total[np.abs(total[..., 0]) <= 1e-8] = 0.0  # the evaluator's rule for negligible functions
            out.append(total)
        return np.concatenate(out, axis=1)

    @staticmethod
    def _center(d, r, shells, values_only):
        i = (r / 0.02).astype(np.int64)
        h = r - i * 0.02
        x, y, z = d.T
        o, zero = np.ones_like(x), np.zeros_like(x)
        angular = ([(o, zero, zero, zero, zero)],
                   [(x, o, zero, zero, zero), (y, zero, o, zero, zero), (z, zero, zero, o, zero)],
                   [(x * x, 2 * x, zero, zero, 2 * o), (y * y, zero, 2 * y, zero, 2 * o), (z * z, zero, zero, 2 * z, 2 * o),
                    (x * y, y, x, zero, zero), (x * z, z, zero, x, zero), (y * z, zero, z, y, zero)])
        cols = []
        for L, c in shells:
            c0, c1, c2, c3 = c[i].T
            f = c0 + h * (c1 + h * (c2 + h * c3))
            fd = (c1 + h * (2 * c2 + 3 * h * c3)) / r
            f2 = 2 * c2 + 6 * h * c3
            for A, ax, ay, az, lap in angular[L]:
                cols.append([A * f] if values_only else
                            [A * f, A * fd * x + ax * f, A * fd * y + ay * f, A * fd * z + az * f,
                             A * f2 + (2 * L + 2) * A * fd + lap * f])
        return np.moveaxis(np.array(cols), -1, 0)

    def _pair(self, r):
        """Cusp function of a pair: value, slope / r, Laplacian."""
        z = r / self.rcut
        p, dp = z - z * z + z ** 3 / 3, 1 - 2 * z + z * z
        q = 1 / (1 + self.gamma * p)
        f = self.rcut * (p * q - 1 / (3 + self.gamma))
        fd = dp * q * q / r
        lap = (-2 + 2 * z) * q * q / self.rcut - 2 * self.gamma * dp * dp * q ** 3 / self.rcut + 2 * fd
        return [np.where(r < self.rcut, self.cusp * v, 0.0) for v in (f, fd, lap)]

    def _single(self, lab, r):
        """One-body function of an atom of this label: value, slope / r, Laplacian."""
        b0, count, rc = self.ei[lab]
        b1 = math.log(b0 + 1.00001)
        out = [0.0, 0.0, 0.0]
        for k, c in enumerate(self.one[lab]):
            b = b0 if k == 0 else math.exp(b1 + 1.6 * k) - 1
            z = r / rc
            p, dp, d2p = z * z * (6 - 8 * z + 3 * z * z), 12 * z * (1 - z) ** 2, 12 * (1 - 4 * z + 3 * z * z)
            q = 1 / (1 + b * p)
            d1 = -(1 + b) * dp * q * q / rc
            d2 = -(1 + b) * (d2p * q * q - 2 * b * dp * dp * q ** 3) / rc ** 2
            for m, v in enumerate(((1 - p) * q, d1 / r, d2 + 2 * d1 / r)):
                out[m] = out[m] + c * np.where(r < rc, v, 0.0)
        return out

    def jastrow_of(self, R, e, p):
        """Terms of electron e[k] placed at p[k] in walker R[k]: value."""
        u = 0.0
        for a, lab in enumerate(self.label):
            u = u + self._single(lab, np.linalg.norm(p - self.at[a], axis=1))[0]
        r = np.linalg.norm(p[:, None] - R, axis=2)
        me = np.arange(self.n)[None] == e[:, None]
        same = (np.arange(self.n)[None] < self.nup) == (e < self.nup)[:, None]
        v = self._pair(np.where(me, 1.0, r))[0] * np.where(same, 0.25, 0.5)
        return u + np.where(me, 0.0, v).sum(1)

    def evaluate(self, R, rot=None):
        w, n = len(R), self.n
        bas = self.basis(R.reshape(-1, 3)).reshape(w, n, -1, 5)
        logpsi, sign = np.zeros(w), np.ones(w)
        gd, ld, inverse = np.zeros((w, n, 3)), np.zeros((w, n)), []
        for s, sl in enumerate((slice(0, self.nup), slice(self.nup, n))):
            phi = np.einsum("wefk,fm->wemk", bas[:, sl], self.mo[:, self.occ[s]], optimize=True)
            if phi.shape[1] == 0:
                inverse.append(None)
                continue
            sg, lg = np.linalg.slogdet(phi[..., 0])
            inv = np.linalg.inv(phi[..., 0])
            d = np.einsum("wemk,wme->wek", phi[..., 1:], inv, optimize=True)
            logpsi, sign = logpsi + lg, sign * sg
            gd[:, sl], ld[:, sl] = d[..., :3], d[..., 3]
            inverse.append(inv)
        gu, lu = np.zeros((w, n, 3)), np.zeros((w, n))
        pot = np.zeros(w)
        for a, lab in enumerate(self.label):
            d = R - self.at[a]
            r = np.sqrt((d * d).sum(2))
            f, fd, lap = self._single(lab, r)
            logpsi, gu, lu = logpsi + f.sum(1), gu + fd[..., None] * d, lu + lap
            pot -= (self.z[a] / r).sum(1)
            pot += sum(self.z[a] * self.z[b] / np.linalg.norm(self.at[a] - self.at[b]) for b in range(a))
        for i in range(n):
            for j in range(i):
                d = R[:, i] - R[:, j]
                r = np.sqrt((d * d).sum(1))
                c = 0.25 if (i < self.nup) == (j < self.nup) else 0.5
                f, fd, lap = (c * v for v in self._pair(r))
                logpsi = logpsi + f
                gu[:, i] += fd[:, None] * d
                gu[:, j] -= fd[:, None] * d
                lu[:, i] += lap
                lu[:, j] += lap
                pot += 1 / r
        lap = ld + lu + (gu * gu).sum(2) + 2 * (gd * gu).sum(2)
        out = dict(logpsi=logpsi, sign=sign, grad=gd + gu, lap=lap, kinetic=-0.5 * lap.sum(1), potential=pot,
                   nonlocal_=np.zeros(w))
        if rot is not None and self.pp:
            out["nonlocal_"] = self._pseudo(R, rot, inverse)
        return out

    def _pseudo(self, R, rot, inverse):
        def channel(terms, r):
            return sum(c * r ** (k - 2) * np.exp(-np.minimum(a * r * r, 60.0)) for k, a, c in terms)

        turn = 2 * math.pi / 10 * np.arange(10)
        c, s = 1 / math.sqrt(5.0), 2 / math.sqrt(5.0)  # the 12 vertices of an icosahedron
        quad = np.array([[0, 0, 1], [0, 0, -1]] + [[s * math.cos(t), s * math.sin(t), c] for t in turn[0::2]] +
                        [[s * math.cos(t), s * math.sin(t), -c] for t in turn[1::2]])
        total = np.zeros(len(R))
        for a, lab in enumerate(self.label):
            if lab not in self.pp:
                continue
            chans = self.pp[lab]
            d = R - self.at[a]
            r = np.sqrt((d * d).sum(2))
            total += channel(chans[-1], r).sum(1)
            # the channels count inside the largest radius (20 bohr down, steps of 0.05) where one is above 1e-5
            grid, at = [], 20.0
            while at > 0:
                grid.append(at)
                at -= 0.05
            cut = max(next((g - 0.05 for g in grid if abs(channel(t, g)) > 1e-5), 20.0) for t in chans[:-1])
            wi, ei = np.nonzero(r < cut)
            ri, di = r[wi, ei], d[wi, ei]
            here = self.jastrow_of(R[wi], ei, R[wi, ei])
            for q in quad:
                u = q @ rot[wi] if rot.ndim == 3 else q @ rot
                p = self.at[a] + u * ri[:, None]
                b = self.basis(p, values_only=True)[..., 0]
                det = np.zeros(len(wi))
                for sp in (0, 1):
                    k = np.flatnonzero((ei >= self.nup) == bool(sp))
                    if len(k):
                        phi = b[k] @ self.mo[:, self.occ[sp]]
                        det[k] = (phi * inverse[sp][wi[k], :, ei[k] - sp * self.nup]).sum(1)
                ratio = det * np.exp(self.jastrow_of(R[wi], ei, p) - here) / 12.0
                cos = (u * di).sum(1) / ri
                v = sum((2 * l + 1) * channel(t, ri) * (1.0, cos)[l] for l, t in enumerate(chans[:-1]))
                np.add.at(total, wi, v * ratio)
        return total


def exact(case, seed):
    if case["call"] in ("vmc", "dmc"):
        return None  # a walk: its random numbers and decisions are the engine's own
    if "cell" in case["system"] and (case["call"] != "orbitals" or case["walkers"] > 1500):
        return None  # a cell's whole wave function (Ewald sums, many images) takes too long this way
    if case["call"] != "orbitals" and case["walkers"] * case["electrons"] ** 2 > 4_000_000:
        return None
    s = prepare(case, seed)
    plain = _Plain(_deck(case))
    if case["call"] == "orbitals":
        R, occ = s["R"], plain.occ[s["spin"]]
        if plain.edge is not None:
            R = R - np.floor(R / plain.edge) * plain.edge
        return dict(rows=np.concatenate([np.einsum("pfk,fm->pmk", plain.basis(p), plain.mo[:, occ], optimize=True)
                                         for p in np.array_split(R, max(1, len(R) // 256))]))
    if case["call"] == "evaluate":
        parts = [plain.evaluate(s["R"][k], s["rot"][k]) for k in np.array_split(np.arange(len(s["R"])), max(1, len(s["R"]) // 128))]
        return {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}
    moved = s["R"].copy()
    k = np.arange(len(moved))
    moved[k, s["electron"]] = s["to"]
    old, new = plain.evaluate(s["R"]), plain.evaluate(moved)
    return dict(dlogpsi=new["logpsi"] - old["logpsi"], sign=new["sign"] * old["sign"], grad=new["grad"][k, s["electron"]],
                lap=new["lap"][k, s["electron"]])
