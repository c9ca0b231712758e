"""Routes of the analyses and the adjoint that depend on sizes or memory: S(q) by runs of q-vectors or one by
one, the RDF's rows of cells, the adjoint with every state kept or recomputed from checkpoints."""
import numpy as np
import pytest

from gamdpy_b200 import _lib, adjoint, workloads

pytestmark = pytest.mark.gpu


def _octant(m):
    n = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[1:]
    return n[(n * n).sum(1) < m * m]


def _sets():
    rng = np.random.default_rng(5)
    line = np.zeros((40, 3), int)
    for axis, name in enumerate("xyz"):
        one = line.copy()
        one[:, axis] = np.arange(-20, 20)
        yield "line_" + name, one
    yield "octant", _octant(9)
    yield "octant_shuffled_twice", rng.permutation(np.concatenate([_octant(7), _octant(7)]))
    yield "slab", np.stack(np.meshgrid(np.arange(-3, 4), [2], np.arange(5, 22), indexing="ij"), -1).reshape(-1, 3)
    yield "one", np.array([[1, -2, 3]])
    yield "sparse", rng.integers(-12, 13, size=(300, 3))
    yield "wide", np.stack([np.arange(600), np.zeros(600, int), np.arange(600) % 2], 1)
    yield "more_than_a_block", _octant(24)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n", [1, 33, 3001])
@pytest.mark.parametrize("name", [k for k, _ in _sets()])
def test_sq_sets_of_q_vectors(name, n, weighted):
    """Runs along each axis, an odd start, duplicates, single and scattered q-vectors, a particle number that
    leaves a partial tile; against float64.  Bound: the phase of a component k is exact to 2 pi |k| 2^-24 in
    float32 (|k| <= 600 here: 2.3e-4 at most, 1e-5 at the usual 24), and independent between particles."""
    nv = dict(_sets())[name]
    rng = np.random.default_rng(n)
    box = np.array([9.0, 11.0, 14.0], np.float32)
    r = ((rng.random((n, 3)) - 0.5) * box).astype(np.float32)
    ff = rng.uniform(0.5, 2.0, n).astype(np.float32) if weighted else None
    got = _lib.sq_compute(r, box, nv, ff)
    w = np.ones(n) if ff is None else ff.astype(np.float64)
    phase = 2 * np.pi * (r.astype(np.float64) / box.astype(np.float64)) @ nv.T.astype(np.float64)
    ref = (w[:, None] * np.exp(1j * phase)).sum(0) / np.sqrt(w.sum())
    k = max(24, np.abs(nv).max())
    assert np.abs(got - ref).max() < 2 * np.pi * k * 2.0 ** -24 * 3 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("bins,nt", [(1, 1), (12289, 1), (64, 3)])
@pytest.mark.parametrize("n", [31, 32, 1000, 5000])
def test_rdf_rows_of_uneven_occupation(oracle, n, bins, nt):
    """Units of 32 slots that span many cells, one dense cell, empty rows; shared and global histograms."""
    rng = np.random.default_rng(n + bins)
    L = np.array([20.0, 21.0, 19.5], np.float32)
    r = (rng.random((n, 3)) - 0.5) * L
    r[: n // 3] = r[0] + rng.normal(0, 0.4, (n // 3, 3))  # a cluster
    r[n // 3 : n // 2, 1:] = r[n // 3, 1:]  # a line along x
    r = (r - L * np.round(r / L)).astype(np.float32)
    pt = rng.integers(0, nt, n).astype(np.int32)
    pt[:nt] = np.arange(nt)
    got = _lib.rdf_compute(r, pt, L, nt, bins, r_max=3.1)
    assert np.array_equal(got, oracle.rdf(r, pt, L, bins, fma=1, r_max=3.1)) and got.sum() > 0


@pytest.mark.parametrize("nt,bins", [(65536, 1), (46341, 1), (2, 1 << 30), (1, 2147483647)])
def test_rdf_refuses_histograms_beyond_int(nt, bins):
    r = np.zeros((4, 3), np.float32)
    with pytest.raises(ValueError, match="rdf"):
        _lib.check(_lib.lib().gdb_rdf_compute(4, _lib.ptr(r), _lib.ptr(np.zeros(4, np.int32)),
                                              _lib.ptr(np.ones(3, np.float32)), nt, bins, 0.4,
                                              _lib.ptr(np.zeros(1, np.uint64))), None, "rdf")


@pytest.mark.parametrize("length", [22.0, 40.0])
@pytest.mark.parametrize("step", [-1, 0])
def test_rdf_whole_and_half_cells(oracle, length, step):
    """The last size of whole cells in x and the first of half ones (six a half cell), every coordinate once on a face;
    a grid just wide enough for plain differences and a wider one."""
    L = np.full(3, length, np.float32)
    edges = float(L[0]) / (3.1 * (1.0 + 1e-4))
    n = 6 * int(2 * edges) * int(edges) ** 2 + step
    rng = np.random.default_rng(n)
    r = ((rng.random((n, 3)) - 0.5) * L).astype(np.float32)
    h = np.float32(0.5) * L[0]
    faces = np.array([h, -h, np.nextafter(h, np.float32(0)), np.nextafter(-h, np.float32(0))], np.float32)
    for axis in range(3):
        r[100 * axis : 100 * (axis + 1), axis] = np.tile(faces, 25)
    pt = rng.integers(0, 2, n).astype(np.int32)
    got = _lib.rdf_compute(r, pt, L, 2, 100, r_max=3.1)
    assert np.array_equal(got, oracle.rdf(r, pt, L, 100, fma=1, r_max=3.1)) and got.sum() > 0


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_rdf_coordinates_on_the_faces(oracle, axis):
    """Particles on the faces of the box and one float away from them, in a grid that takes plain differences."""
    rng = np.random.default_rng(axis)
    L = np.array([22.0, 23.0, 24.0], np.float32)
    r = ((rng.random((4000, 3)) - 0.5) * L).astype(np.float32)
    h = np.float32(0.5) * L[axis]
    faces = np.array([h, -h, np.nextafter(h, np.float32(0)), np.nextafter(-h, np.float32(0))], np.float32)
    r[:400, axis] = np.tile(faces, 100)
    pt = rng.integers(0, 2, 4000).astype(np.int32)
    got = _lib.rdf_compute(r, pt, L, 2, 100, r_max=3.1)
    assert np.array_equal(got, oracle.rdf(r, pt, L, 100, fma=1, r_max=3.1)) and got.sum() > 0


@pytest.mark.parametrize("n,every", [(256, 7), (301, 40), (700, 1)])
def test_adjoint_kept_states_equal_checkpoints(monkeypatch, n, every):
    """Every state kept against segments recomputed from checkpoints: the same numbers, bit for bit."""
    conf = workloads.ka_configuration(n, rho=1.2 if n > 256 else 0.4, temperature=0.6, seed=n)
    cut = np.minimum(workloads.KA_CUT, 0.49 * float(conf.simbox.lengths.min()))
    rdf = {"bins": 12, "r_lo": 0.7, "r_hi": 1.9, "width": 0.1, "every": 3}
    theta = adjoint.theta_from_tables(workloads.KA_SIGMA, workloads.KA_EPSILON)
    out = []
    for keep in (None, "0"):
        if keep is not None:
            monkeypatch.setenv("GDB_ADJ_KEEP_BYTES", keep)
        eng = adjoint.AdjointNVE(conf, cut, dt=0.004, steps=23, checkpoint_every=every, rdf=rdf)
        obs = eng.forward(theta)
        out.append((obs, eng.backward(np.linspace(0.5, 1.5, len(obs))), *eng.final_state()))
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)


def test_adjoint_long_columns_keep_their_order(monkeypatch):
    """A cutoff near half the box: list columns of more than 64 entries, most lanes' hits and skin entries on both sides
    of that boundary.  Segments of 11 steps rebuild their lists at other steps than the kept states' sweep; the sums
    are the same, bit for bit."""
    conf = workloads.lj_configuration([10, 10, 10], 0.85, 2.0, seed=3)
    conf.randomize_velocities(temperature=2.0, seed=3)
    theta = adjoint.theta_from_tables([[1.0]], [[1.0]])
    out = []
    for keep in (None, "0"):
        if keep is not None:
            monkeypatch.setenv("GDB_ADJ_KEEP_BYTES", keep)
        eng = adjoint.AdjointNVE(conf, [[8.2]], dt=0.004, steps=60, checkpoint_every=11)
        obs = eng.forward(theta)
        out.append((obs, eng.backward(np.array([0.5, 1.0, 1.5])), *eng.final_state()))
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)


def test_analyses_from_several_threads():
    """Threads whose calls need different amounts of shared memory of the same kernels: every call succeeds and gives
    what it gives alone."""
    import threading
    rng = np.random.default_rng(8)
    L = np.array([10.0, 10.0, 10.0], np.float32)
    r = ((rng.random((200, 3)) - 0.5) * L).astype(np.float32)
    pt = np.zeros(200, np.int32)
    scattered = rng.integers(-20, 21, size=(40, 3))
    pairs = [(lambda: _lib.sq_compute(r, L, _octant(4)), lambda: _lib.sq_compute(r, L, _octant(16))),
             (lambda: _lib.sq_compute(r, L, scattered % 7), lambda: _lib.sq_compute(r, L, scattered)),
             (lambda: _lib.rdf_compute(r, pt, L, 1, 20), lambda: _lib.rdf_compute(r, pt, L, 1, 9000)),
             (lambda: _lib.rdf_compute(r, pt, L, 1, 20, r_max=2.0), lambda: _lib.rdf_compute(r, pt, L, 1, 9000, r_max=2.0))]
    for pair in pairs:
        wrong = []

        def work(f, want):
            for _ in range(1000):
                try:
                    got = f()
                    if np.abs(got.astype(complex) - want).max() > 1e-9:
                        wrong.append("other numbers")
                except Exception as e:
                    wrong.append(e)

        threads = [threading.Thread(target=work, args=(f, f().astype(complex))) for f in pair for _ in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not wrong, (len(wrong), wrong[:3])
