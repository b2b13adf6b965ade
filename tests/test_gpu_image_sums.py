"""Dispatch edges of the periodic image sums, the e-e-n tables and the warp
teams of the HBM-resident kernels.

* S and P shells of a center sum in registers, four of each shape at a time,
  whatever their order in the deck; a center with a D shell keeps the general
  sums.  Rows against the oracle (1e-10, the FP64 bound of the parity tests);
  quadrature points against single-electron ratios, which use the rows.
* The e-e-n tables hold up to 12 atoms in range per position; more take the
  general routine.
* Results do not depend on the number of warps that share a walker, which the
  walker count decides: sums over the warps only change order (1e-11).
"""
import os
import re

import numpy as np
import pytest

from conftest import GOLDEN
import qworacle
from mainline_b200 import engine, systems

pytestmark = pytest.mark.gpu

# 13 functions per atom each, as the deck's orbital file has them
SHELLS = {"interleaved": ["P", "S", "P", "S", "S", "P", "S"], "many_s": ["S"] * 7 + ["P"] * 2, "one_p": ["S"] * 10 + ["P"],
          "many_p": ["P"] * 4 + ["S"], "d": ["S", "6D", "P", "P"]}


def _rel(a, b):
    return float(np.max(np.abs(a - b) / np.maximum(1.0, np.abs(b))))


def _cell(tmp, shells):
    d = systems.write_periodic(str(tmp), seed=21, name="cell")
    rng = np.random.default_rng(5)
    body = []
    for sym in shells:
        body.append(f"{sym} 2")
        for k in range(2):
            body.append(f"  {k + 1} {rng.uniform(0.15, 4.0)!r} {rng.uniform(0.1, 1.0)!r}")
    text = re.sub(r"GAMESS \{[^}]*\}", "GAMESS {\n" + "\n".join(body) + "\n}", open(d.path).read())
    open(d.path, "w").write(text)
    return d


@pytest.mark.parametrize("kind", list(SHELLS))
def test_rows_and_points_for_every_shell_order(kind, tmp_path):
    d = _cell(tmp_path, SHELLS[kind])
    S = qworacle.System(d.path)
    E = engine.Engine(d.path, engine.FP64, max_walkers=2048)
    P = systems.random_configs(d, 1, seed=4)[0]
    ref = S.mo_lap(P)
    for s, cols in ((0, slice(0, d.nup)), (1, slice(d.nup, d.nelec))):
        assert _rel(E.mo_eval(P, s), ref[:, cols]) < 1e-10
    # nonlocal energy of one walker from the ratios of its quadrature points
    R = P[None]
    rot = systems.random_rotation(np.random.default_rng(8))
    E.set_walkers(R)
    got = E.eval(rot[None]).nonlocal_[0]
    el, to, weight, local = [], [], [], 0.0
    for a, lab in enumerate(S.labels):
        p = S.pp[lab]
        dist = S.min_image(R - S.atoms[a])[0]
        r = np.sqrt((dist ** 2).sum(1))
        vl = [v[0] for v in S._vl_spin(p, r[None], a)]
        local += vl[-1].sum()
        q = p["quad"] @ rot
        for e in np.flatnonzero(r < p["cutoff"]):
            cos = q @ dist[e] / r[e]
            for k in range(len(q)):
                el.append(e)
                to.append(P[e] + q[k] * r[e] - dist[e])
                weight.append(p["w"][k] * sum((2 * l + 1) * vl[l][e] * qworacle.legendre(cos[k], l) for l in range(len(vl) - 1)))
    E.set_walkers(np.repeat(R, len(el), axis=0))
    dl, sg, _, _ = E.ratio(np.array(el), np.array(to))
    terms = np.array(weight) * sg * np.exp(dl)
    assert abs(got - local - terms.sum()) < 1e-10 * (abs(local) + np.abs(terms).sum())
    E.close()


@pytest.mark.parametrize("rcut", [3.3, 6.0])
def test_mixed_move_ratios_with_and_without_the_tables(rcut, tmp_path):
    """e-e-n terms of a 32-atom cell in mixed precision (3.3 bohr: the tables;
    6 bohr: more than 12 atoms in range) against FP64.  The terms are FP64 in
    both, so a wrong one would show at its own size (1e-2 and more); the FP32
    orbitals leave 1e-4 of the ratio away from nodes (the median here)."""
    d = systems.write_periodic(str(tmp_path), seed=13, name="cell", supercell=(2, 2, 1))
    text = open(d.path).read()
    open(d.path, "w").write(text.replace("RCUT 3.3", f"RCUT {rcut}"))
    R = systems.random_configs(d, 32, seed=6)
    rng = np.random.default_rng(7)
    e = rng.integers(0, d.nelec, 32)
    to = R[np.arange(32), e] + rng.normal(0.0, 0.3, (32, 3))
    out = []
    for prec in (engine.FP64, engine.MIXED):
        E = engine.Engine(d.path, prec, max_walkers=32)
        E.set_walkers(R)
        out.append(E.ratio(e, to))
        E.close()
    (d64, _, g64, l64), (dmx, _, gmx, lmx) = out
    assert np.median(np.abs(d64 - dmx)) < 1e-4
    assert np.median(np.abs(g64 - gmx) / (1.0 + np.abs(g64))) < 1e-4
    assert np.median(np.abs(l64 - lmx) / (1.0 + np.abs(l64))) < 1e-3


@pytest.mark.parametrize("name", ["diamond8", "diamond8_k", "mol43"])
def test_evaluation_does_not_depend_on_the_team(name):
    """1 and 592 walkers run on four warps each, 593 and 1200 on two."""
    deck = os.path.join(GOLDEN, name + ".qw")
    d = systems.read_deck(deck)
    R = systems.random_configs(d, 1200, seed=9)
    rot = np.stack([systems.random_rotation(np.random.default_rng(i)) for i in range(1200)])
    E = engine.Engine(deck, engine.FP64, max_walkers=1200)
    E.set_walkers(R)
    ref = E.eval(rot)
    for n in (1, 592, 593):
        E.set_walkers(R[:n])
        ev = E.eval(rot[:n])
        for k in ("logpsi", "grad", "lap", "kinetic", "potential", "nonlocal_"):
            assert _rel(getattr(ev, k), getattr(ref, k)[:n]) < 1e-11, k
    if name != "diamond8_k":
        E.set_walkers(R)
        m0, p0 = E.tmove_select(2, 0.05, seed=3, rot=rot)
        E.set_walkers(R[:5])
        m1, p1 = E.tmove_select(2, 0.05, seed=3, rot=rot[:5])
        assert np.array_equal(m0[:5], m1) and np.allclose(p0[:5], p1, rtol=0, atol=1e-12)
    E.close()
