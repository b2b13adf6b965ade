"""The fused step kernel (VMC blocks, QWG_DMC_SCHEDULE=fused) and the
shared-memory kernels on periodic cells."""
import hashlib
import os
import re

import numpy as np
import pytest

from conftest import GOLDEN
from mainline_b200 import engine, systems
from test_gpu_image_sums import SHELLS, _cell, _rel

pytestmark = pytest.mark.gpu


def _s_first(tmp, d, shells):
    """The deck's trial function with the S shells of every atom listed first."""
    text = open(d.path).read()
    head, orb = open(d.orb_path).read().split("COEFFICIENTS")
    body = re.search(r"GAMESS \{([^}]*)\}", text).group(1).strip().split("\n")
    prims, funcs, f = [], [], 0
    for k, sym in enumerate(shells):
        n = systems.SHELL_NFUNC[sym]
        prims.append(body[3 * k:3 * k + 3])
        funcs.append(list(range(f, f + n)))
        f += n
    order = sorted(range(len(shells)), key=lambda k: shells[k] != "S")
    coef = np.array(orb.split()).reshape(-1, f)[:, sum((funcs[k] for k in order), [])]
    path = str(tmp / "s_first.qw")
    open(str(tmp / "s_first.orb"), "w").write(head + "COEFFICIENTS\n" + "\n".join(" ".join(row) for row in coef) + "\n")
    text = re.sub(r"GAMESS \{[^}]*\}", "GAMESS {\n" + "\n".join("\n".join(prims[k]) for k in order) + "\n}", text)
    open(path, "w").write(text.replace(os.path.basename(d.orb_path), "s_first.orb"))
    return path


@pytest.mark.parametrize("family", ["hbm", "smem"])
@pytest.mark.parametrize("kind", ["interleaved", "many_p", "dropped_s"])
def test_fused_steps_do_not_depend_on_the_shell_order(kind, family, tmp_path, monkeypatch):
    """One VMC step (default depth) and one fused DMC step from the same
    walkers, on a deck that lists P shells first and on the same trial
    function with S first.  The walks are the same up to the order of the
    sums over basis functions (1e-15 a term, a step grows it by less than
    1e4), so energies agree to 1e-9."""
    shells = ["S", "P", "S", "P", "S", "S", "P"] if kind == "dropped_s" else SHELLS[kind]
    d = _cell(tmp_path, shells)
    if kind == "dropped_s":  # the first S shell has no coefficients and is left out of the evaluation
        head, orb = open(d.orb_path).read().split("COEFFICIENTS")
        coef = np.array(orb.split()).reshape(-1, 13)
        coef[:, 0] = "0.0"
        open(d.orb_path, "w").write(head + "COEFFICIENTS\n" + "\n".join(" ".join(row) for row in coef) + "\n")
    if family == "smem":
        monkeypatch.setenv("QWG_KERNEL_FAMILY", "smem")
    monkeypatch.setenv("QWG_DMC_SCHEDULE", "fused")
    R = systems.random_configs(d, 64, seed=14)
    out = []
    for path in (d.path, _s_first(tmp_path, d, shells)):
        E = engine.Engine(path, engine.FP64, max_walkers=64)
        E.set_walkers(R)
        E.vmc_block(1, 0.3, seed=5, deterministic_pp=True)
        got = [E.get_walkers(), E.last_energies()]
        E.set_walkers(R)
        E.dmc_init(0.005, nstep=1, seed=6, deterministic_pp=True)
        E.dmc_block()
        out.append(got + [E.get_walkers(), E.last_energies()])
        E.close()
    for a, b in zip(*out):
        assert _rel(a, b) < 1e-9


def test_vmc_walk_of_a_cell_keeps_its_bits():
    """Three VMC steps (FP64, e-e-n Jastrow, fused step kernel) against walkers
    stored when the walk was pinned.  The orbital tables come from the host's
    exp, so the stored walk holds where the tables are bit for bit the same."""
    deck = os.path.join(GOLDEN, "diamond8.qw")
    g = np.load(os.path.join(GOLDEN, "vmc_walk_cell.npz"))
    h = hashlib.sha256()
    for k in range(engine.inspect_deck(deck).nshell):
        h.update(engine.inspect_spline(deck, k)[0].tobytes())
    if h.hexdigest() != str(g["tables"]):
        pytest.skip("this host's exp gives other orbital tables")
    E = engine.Engine(deck, engine.FP64, max_walkers=16)
    E.set_walkers(g["R0"])
    E.vmc_block(3, 0.3, seed=5)
    assert np.array_equal(E.get_walkers(), g["R"])
    E.close()
