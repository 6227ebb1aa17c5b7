"""On-chip runs of the elastic step (many steps in one launch, one tile of the grid per CTA).

Tiles meet at their halos, at the periodic seam (columns 0 and My, on M- and N-type grids) and at
the x ends, so the grids put few and many tiles of even and odd widths next to each: one tile, the
least tile of 8 rows or columns, tiles whose last vector is partly owned (My mod 4 = 0..3), more rows
than a CTA steps at once, coefficients too many for shared memory. Every field carries random data, the
source sits on a tile edge, receivers on tile edges, the seam and the ends. Fields, residuals and traces
equal the C restatement and the one-step kernels (TW_RESIDENT=0) bit for bit, in one call and in
several; energies to 1e-12 (FP64 sums in another order).
"""
import numpy as np
import pytest

from cases import acoustic_periodic_case, elastic_case, product_acoustic_periodic, product_elastic
from oracle import oracle as orc
from test_tma_gpu import _rcv

pytestmark = pytest.mark.gpu


def _case(Mx, My, cpst, Nt, src_grid="MM"):
    den = max(Mx, My)
    rows, cols = sorted({0, 3, 7, 8, Mx // 2, Mx - 9, Mx - 1}), sorted({0, 1, 7, 8, My // 2, My - 4, My - 1})
    rcvs = [_rcv(tx, ty, r, c, den) for k, (r, c) in enumerate((r, c) for r in rows for c in cols)
            for tx, ty in (("M", "M"), ("N", "M"), ("M", "N"), ("N", "N"))[k % 4:k % 4 + 2]]
    rcvs += [_rcv("N", "N", Mx, My, den), _rcv("M", "N", Mx // 2, My, den), _rcv("N", "M", Mx, 2, den)]
    src = _rcv(src_grid[0], src_grid[1], Mx // 2, 0 if src_grid[1] == "M" else 8, den)
    return elastic_case(Mx, My, seed=Mx + 7 * My, cpst=cpst, Nt=Nt, rcvs=rcvs, src=src, den_dx=den)


def _state(Mx, My, scale=1e-2):
    rng = np.random.default_rng(Mx * My)
    shapes = [(Mx + 1, My + 1), (Mx, My + 1), (Mx + 1, My), (Mx, My), (Mx, My)]
    return [(rng.standard_normal(s) * scale).astype(np.float32).astype(np.float64) for s in shapes]


def _same(got, want, energy):
    for k, v in got["fields"].items():
        assert np.array_equal(v, want["fields"][k]), k
    assert np.array_equal(got["traces"], want["traces"])
    if got["resid"] is not None:
        for a, b in zip(got["resid"], want["resid"]):
            assert np.array_equal(a, b)
    if energy:
        for k in ("E_k", "E_p0", "E_p1"):
            assert np.abs(got[k] - want[k]).max() <= 1e-12 * np.abs(want[k]).max(), k


GRIDS = [(24, 20, (1, 1)), (24, 21, (3, 1)), (25, 22, (1, 2)), (40, 35, (5, 4)), (33, 64, (2, 8)), (97, 61, (1, 2)),
         (150, 90, (2, 2)), (64, 57, (2, 1)), (130, 171, None)]


@pytest.mark.parametrize("cpst,energy", [("00", False), ("00", True), ("3C", False), ("3R", True), ("6C", True), ("6R", False)])
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("Mx,My,tiles", GRIDS)
def test_on_chip_run_matches_restatement_and_single_steps(Mx, My, tiles, prec, cpst, energy, monkeypatch):
    case = _case(Mx, My, cpst, 6, "MM" if energy else "NM")
    f0 = _state(Mx, My)
    r0 = [a * 1e-6 for a in _state(Mx, My)] if cpst != "00" else None
    if tiles is not None:
        monkeypatch.setenv("TW_RES_NTX", str(tiles[0]))
        monkeypatch.setenv("TW_RES_NTY", str(tiles[1]))
    got = product_elastic(case, prec, fields0=f0, resid0=r0, energy=energy)
    monkeypatch.setenv("TW_RESIDENT", "0")
    one = product_elastic(case, prec, fields0=f0, resid0=r0, energy=energy)
    _same(got, one, energy)
    want = orc.elastic_run(case, prec, fields0=f0, **({"resid0": r0} if r0 is not None else {}))
    for k, v in got["fields"].items():
        assert np.array_equal(v, want.fields[k]), k
    assert np.array_equal(got["traces"], want.traces)


@pytest.mark.parametrize("Mx,My,prec", [(700, 701, "f32"), (1000, 1027, "f32"), (600, 803, "f64")])
def test_large_tiles_match_single_steps(Mx, My, prec, monkeypatch):
    """More rows than a CTA steps at once, coefficients kept in L2, and traces of a run in one piece."""
    case = _case(Mx, My, "00", 5)
    f0 = _state(Mx, My)
    got = product_elastic(case, prec, fields0=f0)
    monkeypatch.setenv("TW_RESIDENT", "0")
    _same(got, product_elastic(case, prec, fields0=f0), True)


def test_runs_in_several_calls_and_after_a_reset(tw, monkeypatch):
    """Calls of any length, single steps between them and a second run after a reset (the exchange
    buffer then holds words of the first) give the state and traces of one call."""
    Mx, My = 60, 75
    case = _case(Mx, My, "00", 20)

    def run(calls, resets=0):
        s = tw.Solver(Mx, My, case.num_dx, case.den_dx, case.dt, precision="f32", central_f=case.central_f,
                      time_delay=case.time_delay, max_steps=20, energy=True)
        shp = (Mx + 2, My + 2)
        s.set_material_model(case.rho.reshape(shp), case.vp.reshape(shp), case.vs.reshape(shp))
        s.set_source_location(*case.src)
        for r in case.rcvs:
            s.add_receiver_location(*r)
        for k in range(resets + 1):
            s.reset()
            for n in calls:
                s.step(n)
            s.sync()
        out = ([s.read_field(g, f) for g, f in ((tw.NN, 0), (tw.MN, 0), (tw.NM, 0), (tw.MM, 0), (tw.MM, 1))],
               s.read_receivers(), s.read_energy())
        s.close()
        return out

    want = run([20])
    assert np.abs(want[1]).max() > 0
    for calls, resets in (([1] * 20, 0), ([7, 1, 12], 2), ([20], 1)):
        got = run(calls, resets)
        for a, b in zip(got[0], want[0]):
            assert np.array_equal(a, b)
        assert np.array_equal(got[1], want[1])
        for a, b in zip(got[2], want[2]):
            assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


def test_a_value_that_is_not_finite_is_reported(tw):
    s = tw.Solver(60, 75, 1, 75, 1e-3, precision="f32", max_steps=8, energy=False)
    rng = np.random.default_rng(1)
    s.set_material_model(rng.uniform(1.8, 2.7, (62, 77)), rng.uniform(1.5, 4.5, (62, 77)), rng.uniform(1., 2., (62, 77)))
    f = np.zeros((60, 75))
    f[31, 40] = np.inf
    s.write_field(tw.MM, 0, f)
    with pytest.raises(tw.TwError) as e:
        s.run(3)
    assert e.value.name == "TW_ERR_NONFINITE"
    s.reset()
    s.run(3)
    assert not s.read_field(tw.MM).any()
    s.close()


AC_GRIDS = [(24, 20, (1, 1)), (24, 21, (3, 1)), (25, 22, (1, 2)), (40, 35, (5, 4)), (97, 61, (1, 2)), (64, 57, (2, 1)), (130, 171, None)]


@pytest.mark.parametrize("cpst", ["0", "3", "6"])
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("Mx,My,tiles", AC_GRIDS)
def test_acoustic_periodic_run(Mx, My, tiles, prec, cpst, monkeypatch):
    case = acoustic_periodic_case(Mx, My, seed=Mx + My, cpst=cpst, Nt=7)
    rng = np.random.default_rng(Mx * My)
    f0 = [rng.standard_normal(s).astype(np.float32).astype(np.float64) for s in ((Mx + 1, My), (Mx, My + 1), (Mx, My))]
    r0 = [a * 1e-6 for a in f0] if cpst != "0" else None
    if tiles is not None:
        monkeypatch.setenv("TW_RES_NTX", str(tiles[0]))
        monkeypatch.setenv("TW_RES_NTY", str(tiles[1]))
    got = product_acoustic_periodic(case, prec, fields0=f0, resid0=r0, energy=False)
    monkeypatch.setenv("TW_RESIDENT", "0")
    one = product_acoustic_periodic(case, prec, fields0=f0, resid0=r0, energy=False)
    two = product_acoustic_periodic(case, prec, fields0=f0, resid0=r0, energy=True)   # the two-launch kernels
    for k, v in got["fields"].items():
        assert np.array_equal(v, one["fields"][k]) and np.array_equal(v, two["fields"][k]), k
    assert np.array_equal(got["traces"], one["traces"]) and np.array_equal(got["traces"], two["traces"])
    for a, b in zip(got.get("resid") or [], one.get("resid") or []):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("cpst", ["00", "3C", "3R", "6C", "6R"])
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("Mx,My,tiles", AC_GRIDS)
def test_acoustic_free_surface_run(Mx, My, tiles, prec, cpst, monkeypatch):
    """These handles hold one copy of the state: a run ends in the buffer it began in."""
    den = max(Mx, My)
    rcvs = [_rcv("M", "M", r, c, den) for r in (0, 8, Mx - 1) for c in (0, 8, My - 1)]
    case = elastic_case(Mx, My, seed=5, cpst=cpst, Nt=7, rcvs=rcvs, den_dx=den, acoustic=True)
    rng = np.random.default_rng(Mx * My)
    f0 = [rng.standard_normal(s).astype(np.float32).astype(np.float64) for s in ((Mx, My + 1), (Mx + 1, My), (Mx, My))]
    if tiles is not None:
        monkeypatch.setenv("TW_RES_NTX", str(tiles[0]))
        monkeypatch.setenv("TW_RES_NTY", str(tiles[1]))
    got = product_elastic(case, prec, acoustic=True, fields0=f0, energy=False)
    monkeypatch.setenv("TW_RESIDENT", "0")
    one = product_elastic(case, prec, acoustic=True, fields0=f0, energy=False)
    _same(got, one, False)


@pytest.mark.parametrize("bc", ["periodic", "free"])
def test_acoustic_runs_in_several_calls_and_in_a_batch(tw, bc, monkeypatch):
    """Single steps, runs and batch steps mixed on the same handles equal the per-point kernels."""
    Mx, My = 60, 75

    def run(calls, resident, batch_at=None):
        monkeypatch.setenv("TW_RESIDENT", "1" if resident else "0")
        shots = []
        for k in range(2):
            s = tw.Solver(Mx, My, 1, My, 1e-3, physics=tw.ACOUSTIC, bc_x=tw.PERIODIC if bc == "periodic" else tw.SAT_FREE,
                          precision="f32", max_steps=40, energy=False)
            rng = np.random.default_rng(k)
            s.set_material_grid(tw.NM, 0, rng.uniform(1, 2, (Mx + 1, My)))
            s.set_material_grid(tw.MN, 0, rng.uniform(1, 2, (Mx, My + 1)))
            s.set_material_grid(tw.MM, 0, rng.uniform(1, 2, (Mx, My)))
            s.set_source(tw.NM if bc == "periodic" else tw.MM, 1, 1)
            s.add_receivers(tw.MM, [0, 30, 59], [0, 8, 74])
            s.write_field(tw.MM, 0, rng.standard_normal((Mx, My)))
            shots.append(s)
        b = tw.Batch(shots)
        for i, n in enumerate(calls):
            if i == batch_at:
                b.step(3)
            for s in shots:
                s.step(n)
        b.sync()
        out = [[s.read_field(g) for g in (tw.MN, tw.NM, tw.MM)] + [s.read_receivers()] for s in shots]
        b.close()
        for s in shots:
            s.close()
        return out

    for calls, at in (([20], None), ([1, 7, 2, 1, 6], None), ([5, 1, 8], 1), ([4, 4], 1)):
        for x, y in zip(run(calls, True, at), run(calls, False, at)):
            for p, q in zip(x, y):
                assert np.array_equal(p, q), (calls, at)


def test_handles_of_different_sizes_side_by_side(tw):
    """Handles share the kernels: one made later, smaller, must not take shared memory from another."""
    sizes = [(300, 330), (24, 20), (700, 640), (40, 60)]
    shots = []
    for Mx, My in sizes:
        s = tw.Solver(Mx, My, 1, My, 1e-4, precision="f32", max_steps=8, energy=False)
        rng = np.random.default_rng(Mx)
        P = (Mx + 2, My + 2)
        s.set_material_model(rng.uniform(1.8, 2.7, P), rng.uniform(1.5, 4.5, P), rng.uniform(1., 2., P))
        s.write_field(tw.MM, 0, rng.standard_normal((Mx, My)))
        shots.append(s)
    alone = []
    for s in shots:
        s.run(4)
        alone.append(s.read_field(tw.MM, 0))
    assert all(np.isfinite(a).all() and np.abs(a).max() > 0 for a in alone)
    for s in shots:   # queued together, on a stream each
        s.step(2)
    for s in shots:
        s.step(2)
    for s in shots:
        s.sync()
        s.close()


@pytest.mark.parametrize("bc,prec,cpst", [("periodic", "f32", "00"), ("periodic", "f64", "3R"), ("periodic", "f32", "6R"),
                                          ("free", "f32", "00"), ("free", "f64", "6R")])
def test_batch_on_chip_matches_the_batch_kernels(tw, bc, prec, cpst, monkeypatch):
    """Shots of uneven sizes that all fit on the chip step in groups of tiles; more than one group here."""
    sizes = [(8, 8), (20, 33), (300, 300), (257, 511), (400, 420), (61, 700), (330, 340), (500, 380), (1000, 1030)]

    def run(resident):
        monkeypatch.setenv("TW_RESIDENT", "1" if resident else "0")
        shots = []
        for k, (Mx, My) in enumerate(sizes):
            s = tw.Solver(Mx, My, 1, My, 1e-4, physics=tw.ACOUSTIC, bc_x=tw.PERIODIC if bc == "periodic" else tw.SAT_FREE,
                          precision=prec, cpst=cpst, max_steps=16, energy=False)
            rng = np.random.default_rng(k)
            for g in (tw.NM, tw.MN, tw.MM):
                s.set_material_grid(g, 0, rng.uniform(1, 2, s.shape(g)))
                s.write_field(g, 0, rng.standard_normal(s.shape(g)))
            s.set_source(tw.MM, Mx // 2, My // 2)
            s.add_receivers(tw.MM, [0, Mx // 2, Mx - 1], [My - 1, My // 2, 0])
            s.add_receivers(tw.NM, [Mx - 1], [1])
            shots.append(s)
        b = tw.Batch(shots)
        for n in (5, 1, 6, 2):
            b.step(n)
        b.sync()
        out = [[s.read_field(g) for g in (tw.MN, tw.NM, tw.MM)] + [s.read_receivers()] for s in shots]
        b.close()
        for s in shots:
            s.close()
        return out

    for k, (x, y) in enumerate(zip(run(True), run(False))):
        assert np.abs(x[3]).max() > 0
        for p, q in zip(x, y):
            assert np.array_equal(p, q), k
