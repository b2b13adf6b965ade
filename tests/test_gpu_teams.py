"""Teams of warps in the HBM-resident kernels, and the tables of the e-e-n terms.

A walker's team has 4 warps up to 592 walkers, 2 below 2368 walkers or from 32
electrons, else 1.  The warps share the terms of its sums, so that only the
order of the sums depends on their number."""
import os
import re

import numpy as np
import pytest

from conftest import GOLDEN
import qworacle
from mainline_b200 import engine, systems
from test_gpu_image_sums import _rel

pytestmark = pytest.mark.gpu


def _molecule(tmp, nelec=20):
    """A molecule of the HBM-resident kernels below 32 electrons, with e-e-n terms."""
    d = systems.write_molecule(str(tmp), "mol", 77, nelec)
    rng = np.random.default_rng(3)
    text = open(d.path).read()
    labels = re.findall(r"EIBASIS \{ (\S+) ", text)
    text = text.replace("  ONEBODY {", "  EEBASIS { EE POLYPADE BETA0 0.5 NFUNC 3 RCUT 7.5 }\n  ONEBODY {")
    terms = "\n".join(f"    COEFFICIENTS {{ {a} " + " ".join(map(repr, rng.normal(0, 0.05, 8).tolist())) + " }" for a in labels)
    at = text.rindex("  }\n}\n  }\n}")
    open(d.path, "w").write(text[:at] + "  }\n  THREEBODY {\n" + terms + "\n" + text[at:])
    return d


@pytest.mark.parametrize("prec", [engine.FP64, engine.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", ["mol20", "diamond8", "diamond8_k", "mol43", "n2_multidet"])
def test_results_do_not_depend_on_the_population(name, prec, tmp_path):
    """Evaluations, T-move selections and steps of the split schedule of the
    first walkers of 2400 (one warp each below 32 electrons), 593 (two) and 5 (four)."""
    if name == "mol20":
        d = _molecule(tmp_path)
    else:
        d = systems.read_deck(os.path.join(GOLDEN, name + ".qw"))
    R = systems.random_configs(d, 2400, seed=9)
    rot = np.stack([systems.random_rotation(np.random.default_rng(i)) for i in range(2400)])
    out = []
    for n in (2400, 593, 5):
        E = engine.Engine(d.path, prec, max_walkers=2400)  # the random streams go on with a context's steps
        E.set_walkers(R[:n])
        ev = E.eval(rot[:n])
        got = [getattr(ev, k)[:5] for k in ("logpsi", "sign", "grad", "lap", "kinetic", "potential", "nonlocal_")]
        if name != "diamond8_k":
            for mode in (1, 2):
                got += [x[:5] for x in E.tmove_select(mode, 0.05, seed=3, rot=rot[:n])]
        E.set_vmc_dynamics(depth=1)
        E.set_walkers(R[:n])
        E.vmc_block(2, 0.1, seed=4)
        out.append(got + [E.get_walkers()[:5], E.last_energies()[:5]])
        E.close()
    for other in out[1:]:
        for a, b in zip(out[0], other):  # sums of up to 1e4 FP64 terms below 1e3
            assert _rel(a, b) < 1e-9


def test_tensor_core_rows_do_not_depend_on_the_population(tmp_path, monkeypatch):
    """One step of the tensor-core move schedule: basis rows by two warps
    (1024 walkers) and by one (2400)."""
    monkeypatch.setenv("QWG_TC_MOVES", "1")
    d = _molecule(tmp_path)
    R = systems.random_configs(d, 2400, seed=9)
    out = []
    for n in (2400, 1024):
        E = engine.Engine(d.path, engine.MIXED, max_walkers=2400)
        E.set_vmc_dynamics(depth=1)
        E.set_walkers(R[:n])
        E.vmc_block(1, 0.1, seed=4)
        out.append((E.get_walkers()[:1024], E.last_energies()[:1024]))
        E.close()
    assert np.array_equal(out[0][0], out[1][0])  # moves take no sums over the team
    assert _rel(out[0][1], out[1][1]) < 1e-9


def _cell(tmp, rcut, wide, scale):
    """The 32-atom cell; e-n and e-e-n cutoff rcut, with wide another one-body
    group that reaches beyond it; all their coefficients times scale."""
    d = systems.write_periodic(str(tmp), seed=13, name=f"cell{scale}", supercell=(2, 2, 1))
    head, group = open(d.path).read().rsplit("GROUP {", 1)
    group = group.replace("RCUT 3.3", f"RCUT {rcut}")

    def times(m):
        return m.group(1) + " ".join(repr(scale * float(c)) for c in m.group(2).split()) + " }"

    group = re.sub(r"(COEFFICIENTS \{ X )([^}]*)\}", times, group)
    extra = ("GROUP {\n  EIBASIS { X POLYPADE BETA0 0.9 NFUNC 2 RCUT 3.3 }\n  ONEBODY {\n    COEFFICIENTS { X "
             f"{0.3 * scale!r} {-0.2 * scale!r} }}\n  }}\n}}\n") if wide else ""
    open(d.path, "w").write(head + extra + "GROUP {" + group)
    return d


@pytest.mark.parametrize("rcut,wide", [(3.3, False), (3.0, True), (6.0, False)])
def test_e_e_n_terms_of_mixed_proposals(rcut, wide, tmp_path):
    """Every move's e-n and e-e-n terms in mixed precision (from the tables;
    6 bohr: more atoms in range than they hold) against FP64.  They are FP64 in
    both.  The difference of the deck and of the same deck with zero
    coefficients leaves them alone: the determinant and the pair functions are
    the same numbers in either.  Bounds: 1e-15 a term of a few hundred, with
    the size of what cancels."""
    R = systems.random_configs(_cell(tmp_path, rcut, wide, 1.0), 48, seed=6)
    rng = np.random.default_rng(7)
    e = rng.integers(0, R.shape[1], 48)
    to = R[np.arange(48), e] + rng.normal(size=(48, 3)) * np.repeat([0.05, 0.6, 2.5], 16)[:, None]
    diff = []
    for prec in (engine.FP64, engine.MIXED):
        got = []
        for scale in (1.0, 0.0):
            E = engine.Engine(_cell(tmp_path, rcut, wide, scale).path, prec, max_walkers=48)
            E.set_walkers(R)
            dl, _, g, l = E.ratio(e, to)
            got.append((dl, g, l - (g * g).sum(1), 1.0 + np.abs(l) + (g * g).sum(1)))
            E.close()
        (a, b) = got
        diff.append((a[0] - b[0], a[1] - b[1], a[2] - b[2], a[3] + b[3]))
    (u0, g0, l0, s0), (u1, g1, l1, s1) = diff
    assert np.all(np.abs(u0 - u1) < 1e-11)
    assert np.all(np.abs(g0 - g1) < 1e-11 * (s0 + s1)[:, None])
    assert np.all(np.abs(l0 - l1) < 1e-11 * (s0 + s1))
    assert np.abs(u0).max() > 1e-2


def test_item_list_that_overruns_the_e_n_table(tmp_path):
    """The electrons' e-n values stand at the end of the item list.  With two
    more e-n functions an atom, of zero coefficient, electrons inside three or
    more cutoffs each give more items than that leaves room for; the deck
    without them has room.  Both state the same trial function."""
    d = systems.write_periodic(str(tmp_path), seed=13, name="cell")
    text = open(d.path).read()
    text = text.replace("NFUNC 4 RCUT 3.3", "NFUNC 6 RCUT 3.3")
    text = re.sub(r"(ONEBODY \{\s*COEFFICIENTS \{ X [^}]*)\}", r"\1 0.0 0.0 }", text)
    six = str(tmp_path / "six.qw")
    open(six, "w").write(text)
    S = qworacle.System(d.path)
    cutoff = S.pp[S.labels[0]]["cutoff"]

    def in_range(x):
        return sum((np.linalg.norm(S.min_image(x - a), axis=-1) < cutoff).astype(int) for a in S.atoms)

    rng = np.random.default_rng(2)
    x = rng.uniform(0.0, 6.74, (4000, 3))
    n = in_range(x[None])[0]
    R = np.concatenate([x[n <= 2][:2 * d.nelec], x[n >= 3][:2 * d.nelec]]).reshape(4, d.nelec, 3)
    N, A = d.nelec, d.natoms
    room = [(72 * N * A - N * (8 + A * k * 8)) // 72 for k in (4, 6)]  # 72-byte items, FP64 values
    items = in_range(R).sum(1)
    assert items.max() < room[0] and items[:2].max() < room[1] < items[2:].min()
    rot = np.stack([systems.random_rotation(rng) for _ in R])
    got = []
    for path in (d.path, six):
        E = engine.Engine(path, engine.FP64, max_walkers=4)
        E.set_walkers(R)
        got.append(E.eval(rot).nonlocal_)
        E.close()
    assert _rel(*got) < 1e-10
