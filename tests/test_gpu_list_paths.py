"""Neighbour-list builds over the sizes where the lanes per particle and the launch shape of the persistent
kernel change, against the oracle's sets; pair exclusions on each of them; forces on the same
lists.  Bars: sets bit-exact, forces 1e-5 relative RMS (float32 sums of ~100 terms in another order)."""
import numpy as np
import pytest

from conftest import rel_rms, sorted_rows
from gamdpy_b200 import _lib, workloads
from test_gpu_parity import FORCE_TOL, make_sim

pytestmark = pytest.mark.gpu

SKIN = 0.3
CPS = float(np.float32(2.5) + np.float32(SKIN))


def _table(oracle):
    return oracle.param_table([workloads.KA_SIGMA, workloads.KA_EPSILON, workloads.KA_CUT])


def _reference(oracle, r, L):
    if len(r) <= 20011:
        return oracle.nblist_nsq(r, L, CPS, 300, fma=1)[0]
    return oracle.nblist_cells(r, L, 2.5, SKIN, 300, fma=1)[0]


@pytest.mark.parametrize("n", [3073, 4737, 4738, 10007, 37889, 75777, 151552, 151553, 190001])
@pytest.mark.parametrize("persistent", [True, False])
def test_cell_lists_over_launch_shapes(oracle, n, persistent):
    """Lanes 16 to 1 per particle, the last size with one block per SM and the rounds beyond; a partial last
    warp in each."""
    conf = workloads.ka_configuration(n, seed=n, jitter=0.2)
    L = conf.simbox.lengths
    sim = make_sim(conf["r"], L, conf.ptype, _table(oracle), nblist=_lib.NBLIST_CELLS, skin=SKIN)
    if persistent:
        sim.run(0.0, 0)  # no steps: the evaluation's list, of the uploaded positions
    else:
        sim.eval_forces()
    ref = _reference(oracle, conf["r"], L)
    c1, f1 = sorted_rows(sim.nblist(300))
    c2, f2 = sorted_rows(ref)
    assert np.array_equal(c1, c2) and np.array_equal(f1, f2)
    if not persistent:
        res = oracle.forces(conf["r"], conf.ptype, L, _table(oracle), ref, fma=1)
        assert rel_rms(sim.download()["f"], res["f"]) < FORCE_TOL


@pytest.mark.parametrize("n,kind", [(2050, _lib.NBLIST_NSQ), (3073, _lib.NBLIST_CELLS), (4737, _lib.NBLIST_CELLS),
                                    (10007, _lib.NBLIST_CELLS), (37889, _lib.NBLIST_CELLS),
                                    (75777, _lib.NBLIST_CELLS), (151553, _lib.NBLIST_CELLS)])
def test_lists_with_rounded_products(oracle, n, kind, monkeypatch):
    """GDB_NBLIST_FMA=0: the distances' products rounded before they are added (gamdpy's CPU build), over the lanes per
    particle of the cell build and in the N^2 build."""
    monkeypatch.setenv("GDB_NBLIST_FMA", "0")
    monkeypatch.setenv("GDB_CLUSTER", "0")
    conf = workloads.ka_configuration(n, seed=n, jitter=0.2)
    L = conf.simbox.lengths
    sim = make_sim(conf["r"], L, conf.ptype, _table(oracle), nblist=kind, skin=SKIN)
    sim.run(0.0, 0)
    if n <= 20011:
        ref = oracle.nblist_nsq(conf["r"], L, CPS, 300, fma=0)[0]
    else:
        ref = oracle.nblist_cells(conf["r"], L, 2.5, SKIN, 300, fma=0)[0]
    c1, f1 = sorted_rows(sim.nblist(300))
    c2, f2 = sorted_rows(ref)
    assert np.array_equal(c1, c2) and np.array_equal(f1, f2)


@pytest.mark.parametrize("n", [257, 1024, 1025, 3000])
@pytest.mark.parametrize("persistent", [True, False])
def test_nsq_lists_over_mask_edges(oracle, n, persistent, monkeypatch):
    """1024 candidates fill a warp's masks once; one warp with and one without a second particle."""
    monkeypatch.setenv("GDB_CLUSTER", "0")
    conf = workloads.ka_configuration(n, rho=1.2 if n > 300 else 0.6, seed=n, jitter=0.2)
    L = conf.simbox.lengths
    sim = make_sim(conf["r"], L, conf.ptype, _table(oracle), nblist=_lib.NBLIST_NSQ, skin=SKIN)
    sim.run(0.0, 0) if persistent else sim.eval_forces()
    c1, f1 = sorted_rows(sim.nblist(300))
    c2, f2 = sorted_rows(_reference(oracle, conf["r"], L))
    assert np.array_equal(c1, c2) and np.array_equal(f1, f2)


@pytest.mark.parametrize("n,kind", [(2050, _lib.NBLIST_NSQ), (5001, _lib.NBLIST_CELLS), (160010, _lib.NBLIST_CELLS)])
def test_exclusions_on_every_build(oracle, n, kind):
    """Pairs (i, i + 1) of chains of five excluded: the oracle's list without them."""
    conf = workloads.ka_configuration(n, seed=n, jitter=0.2)
    L = conf.simbox.lengths
    i = np.arange(n)
    excl = np.zeros((n, 3), np.int32)
    for other, ok in ((i + 1, (i % 5 != 4) & (i + 1 < n)), (i - 1, i % 5 != 0)):
        k = excl[ok, 2]
        excl[ok, k] = other[ok]
        excl[ok, 2] = k + 1
    sim = make_sim(conf["r"], L, conf.ptype, _table(oracle), nblist=kind, skin=SKIN)
    sim.set_exclusions(excl)
    sim.run(0.0, 0)
    ref = oracle.exclude(_reference(oracle, conf["r"], L), excl)
    c1, f1 = sorted_rows(sim.nblist(300))
    c2, f2 = sorted_rows(ref)
    assert np.array_equal(c1, c2) and np.array_equal(f1, f2)


@pytest.mark.parametrize("n", [300, 1184, 1185, 1776, 1777, 2048, 10007, 37889])
def test_first_run_through_graphs(oracle, n, monkeypatch):
    """Without the persistent kernel, the first run of a handle captures its steps into a graph, where nothing can be
    allocated; sizes whose standalone step has more lanes than the persistent kernel's, and the lines of that kernel's
    lanes and blocks at small sizes.  Against that kernel after 32
    steps: coordinates to 1e-4 (an ulp of a coordinate here is 1e-6 and either path rounds them 32 times)."""
    conf = workloads.ka_configuration(n, seed=n)
    L = np.asarray(conf.simbox.lengths, np.float32)
    monkeypatch.setenv("GDB_CLUSTER", "0")
    out = []
    for persistent in ("0", "1"):
        monkeypatch.setenv("GDB_PERSISTENT", persistent)
        sim = make_sim(conf["r"], L, conf.ptype, _table(oracle), nblist=_lib.NBLIST_CELLS, skin=SKIN, v=conf["v"])
        sim.set_nvt(0.005, 0.2, _lib.TFUNC_CONSTANT, [0.45])
        sim.run(0.0, 32)
        assert sim.last_path() == int(persistent)
        out.append(sim.download()["r"])
    d = out[0] - out[1]
    d -= L * np.round(d / L)
    assert np.abs(d).max() < 1e-4
