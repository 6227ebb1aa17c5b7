"""Calls around the on-chip runs: waits that give up, short calls, batches whose shots change after
the batch was made, memory kept after a gradient. What runs on the chip is compared with the handle's
other step kernels (TW_RESIDENT=0) bit for bit.
"""
import numpy as np
import pytest

from cases import elastic_case
from test_adjoint_gpu import rcvs_for, solver

pytestmark = pytest.mark.gpu


def test_a_gradient_whose_exchanges_give_up_is_an_error(tw, monkeypatch):
    """With no polls every tile leaves its run at the first exchange: the states are incomplete."""
    case = elastic_case(130, 150, seed=3, Nt=12, den_dx=150, rcvs=rcvs_for(130, 150, 150))
    obs = np.zeros((len(case.rcvs), 2, 12))
    monkeypatch.setenv("TW_RES_POLLS", "0")
    s = solver(tw, case, precision="f32")
    with pytest.raises(tw.TwError) as e:
        s.run(12)
    assert e.value.name == "TW_ERR_TIMEOUT"
    s.reset()
    with pytest.raises(tw.TwError) as e:
        s.adjoint_gradient(12, obs, ckpt_every=5)
    assert e.value.name == "TW_ERR_TIMEOUT"
    s.close()
    monkeypatch.delenv("TW_RES_POLLS")
    s = solver(tw, case, precision="f32")
    assert np.isfinite(s.adjoint_gradient(12, obs, ckpt_every=5)["misfit"])
    s.close()


def test_a_gradient_keeps_a_bounded_amount_of_memory(tw):
    """A gradient whose checkpoints take 5 GB leaves at most 4 GiB with the library, all of it on request."""
    import torch
    M, nt = 2048, 60
    s = tw.Solver(M, M, 1, 500, 1e-4, precision="f32", max_steps=nt, energy=False)
    model = [np.full((M + 2, M + 2), v) for v in (2.0, 3.0, 1.7)]
    s.set_material_model(*model)
    s.set_source(tw.MM, M // 2, M // 2)
    s.add_receivers(tw.NM, [M // 2], [M // 2 + 4])
    obs = np.zeros((1, 2, nt))
    s.adjoint_gradient(2, np.zeros((1, 2, 2)), ckpt_every=1, model=False)   # (kernels loaded, host buffers made)
    s.reset()
    tw.release_cached_memory()
    before = torch.cuda.mem_get_info()[0]
    assert s.adjoint_gradient(nt, obs, ckpt_every=nt, model=False)["misfit"] > 0
    slack = 256 << 20
    assert before - torch.cuda.mem_get_info()[0] <= (4 << 30) + slack
    tw.release_cached_memory()
    assert before - torch.cuda.mem_get_info()[0] <= slack
    s.close()


def acoustic(tw, Mx, My, bc, k=0, max_steps=64, precision="f32", cpst="00"):
    """A shot with random medium and fields, a source and a few receivers."""
    s = tw.Solver(Mx, My, 1, max(Mx, My), 1e-4, physics=tw.ACOUSTIC, bc_x=tw.PERIODIC if bc == "periodic" else tw.SAT_FREE,
                  precision=precision, cpst=cpst, max_steps=max_steps, energy=False)
    rng = np.random.default_rng(k)
    for g in (tw.NM, tw.MN, tw.MM):
        s.set_material_grid(g, 0, rng.uniform(1, 2, s.shape(g)))
        s.write_field(g, 0, rng.standard_normal(s.shape(g)))
    s.set_source(tw.MM, Mx // 2, My // 2)
    s.add_receivers(tw.MM, [0, Mx // 2, Mx - 1], [My - 1, My // 2, 0])
    s.add_receivers(tw.NM, [Mx - 1], [1])
    return s


def result(tw, s):
    return [s.read_field(g) for g in (tw.MN, tw.NM, tw.MM)] + [s.read_receivers()]


def same(a, b):
    return all(np.array_equal(p, q) for x, y in zip(a, b) for p, q in zip(x, y))


@pytest.mark.parametrize("resident", [True, False])
@pytest.mark.parametrize("bc", ["periodic", "free"])
def test_a_batch_takes_up_receivers_and_sources_set_later(tw, bc, resident, monkeypatch):
    """Receivers added between two batch steps (more than the shot's trace buffer held, which moves) and a
    source set anew give what the shots stepped alone give."""
    monkeypatch.setenv("TW_RESIDENT", "1" if resident else "0")
    sizes = [(60, 75), (130, 41)]

    def run(batched):
        shots = [acoustic(tw, Mx, My, bc, k) for k, (Mx, My) in enumerate(sizes)]
        b = tw.Batch(shots) if batched else None

        def step(n):
            if b:
                b.step(n)
            for s in shots if not b else []:
                s.step(n)

        step(10)
        shots[0].add_receivers(tw.MM, np.arange(40), np.arange(40))
        shots[1].add_receivers(tw.MN, [3], [4])
        step(17)
        shots[1].set_source(tw.MN, 7, 9)
        shots[0].clear_source()
        step(18)
        step(1)
        for h in [b] if b else shots:
            h.sync()
        out = [result(tw, s) for s in shots]
        for h in ([b] if b else []) + shots:
            h.close()
        return out

    got, want = run(True), run(False)
    assert np.abs(want[0][3][4:, 0, 10:]).max() > 0 and not want[0][3][4:, 0, :10].any()
    assert same(got, want)


@pytest.mark.parametrize("physics,Mx,My", [("elastic", 890, 884), ("elastic", 886, 884), ("periodic", 128, 61), ("free", 77, 40)])
def test_single_steps_and_runs_in_turn(tw, physics, Mx, My, monkeypatch):
    """Calls of one step go by other kernels than longer ones (elastic: from 3 x 2^18 cells on)."""
    def run(resident):
        monkeypatch.setenv("TW_RESIDENT", "1" if resident else "0")
        if physics == "elastic":
            s = tw.Solver(Mx, My, 1, My, 1e-4, precision="f32", max_steps=16, energy=False)
            rng = np.random.default_rng(1)
            s.set_material_model(*[rng.uniform(a, b, (Mx + 2, My + 2)) for a, b in ((1.8, 2.7), (3., 4.5), (1., 2.))])
            s.write_field(tw.MM, 0, rng.standard_normal((Mx, My)))
            s.set_source(tw.MM, Mx // 2, 0)
            s.add_receivers(tw.NM, [0, Mx // 2, Mx], [My - 1, 3, 0])
        else:
            s = acoustic(tw, Mx, My, physics, max_steps=16)
        for n in (1, 1, 3, 1, 2, 1, 1, 4):
            s.step(n)
        s.sync()
        out = result(tw, s)
        s.close()
        return out

    assert same([run(True)], [run(False)])


@pytest.mark.parametrize("bc", ["periodic", "free"])
@pytest.mark.parametrize("prec,cpst", [("f32", "00"), ("f64", "00"), ("f32", "6R")])
@pytest.mark.parametrize("sizes", [[(61, 70)], [(200, 330)] * 2, [(64, 64), (300, 41), (9, 900)], [(256, 250)] * 5 + [(40, 40)],
                                   [(512, 500)] * 4 + [(100, 90)]])
def test_batches_of_few_shots(tw, sizes, prec, cpst, bc, monkeypatch):
    """Few shots share all the SMs: tilings of more tiles than the least, groups of one shot and of several."""
    def run(resident):
        monkeypatch.setenv("TW_RESIDENT", "1" if resident else "0")
        shots = [acoustic(tw, Mx, My, bc, k, precision=prec, cpst=cpst) for k, (Mx, My) in enumerate(sizes)]
        b = tw.Batch(shots)
        for n in (9, 2, 12):
            b.step(n)
        b.sync()
        out = [result(tw, s) for s in shots]
        for h in [b] + shots:
            h.close()
        return out

    assert same(run(True), run(False))


@pytest.mark.parametrize("bc", ["periodic", "free"])
def test_batch_calls_of_every_length(tw, bc, monkeypatch):
    """Calls too short for a batch of several groups go by the batch kernels, longer ones on chip, in turn."""
    def run(resident):
        monkeypatch.setenv("TW_RESIDENT", "1" if resident else "0")
        shots = [acoustic(tw, 520, 500 + k, bc, k) for k in range(7)]
        b = tw.Batch(shots)
        for n in (1, 7, 2, 3, 6, 4, 1, 5):
            b.step(n)
        b.sync()
        out = [result(tw, s) for s in shots]
        for h in [b] + shots:
            h.close()
        return out

    assert same(run(True), run(False))


def _gives_up(tw, h):
    try:
        h.sync()
    except tw.TwError as e:
        assert e.name == "TW_ERR_TIMEOUT"
        return True
    return False


def test_which_batch_calls_run_on_chip(tw, monkeypatch):
    """With no polls a call of two steps or more that runs on chip times out, and any other does not (one step
    exchanges nothing)."""
    monkeypatch.setenv("TW_RES_POLLS", "0")
    for bc, k, least in (("periodic", 3, 2), ("periodic", 8, 4), ("free", 8, 3), ("periodic", 12, 6), ("free", 12, 4)):
        shots = [acoustic(tw, 512, 512, bc, max_steps=16) for _ in range(k)]
        b = tw.Batch(shots)
        b.step(least - 1)
        assert not _gives_up(tw, b), (bc, k)
        b.step(least)
        assert _gives_up(tw, b), (bc, k)
        for h in [b] + shots:
            h.close()


@pytest.mark.parametrize("bc,shape", [("periodic", (0, 0, 0, 8)), ("free", (64, 4, 2, 0))])
def test_a_launch_shape_that_was_asked_for_is_used(tw, bc, shape, monkeypatch):
    """After tw_batch_set_shape no call runs on chip (where it would time out here), until tw_batch_tune; the shape
    found by tune is the batch kernels'."""
    want = acoustic(tw, 200, 210, bc, max_steps=40)
    want.run(30)
    monkeypatch.setenv("TW_RES_POLLS", "0")
    s = acoustic(tw, 200, 210, bc, max_steps=40)
    b = tw.Batch([s])
    b.set_shape(*shape)
    b.step(30)
    assert not _gives_up(tw, b)
    assert same([result(tw, s)], [result(tw, want)])
    assert b.tune(4) > 0
    assert b.shape()[2] in ((2, 4, 8, 15, 24, 32, 48, 64) if bc == "periodic" else (1, 2, 4))
    b.step(30)
    assert _gives_up(tw, b)
    for h in (b, s, want):
        h.close()


def test_a_handle_without_room_for_the_exchange_words_steps_by_its_other_kernels(tw, monkeypatch):
    """With the GPU's memory all but taken, a handle that would fit without its on-chip buffers (53 MB here) is
    made and steps as one that never had them."""
    import torch
    M = 740

    def run():
        s = tw.Solver(M, M, 1, M, 1e-4, precision="f64", max_steps=8, energy=False)
        s.set_material_model(*[np.full((M + 2, M + 2), v) for v in (2.0, 3.0, 1.7)])
        s.set_source(tw.MM, 300, 300)
        s.run(5)
        out = s.read_field(tw.MM)
        s.close()
        return out

    run()   # (kernels loaded)
    monkeypatch.setenv("TW_RESIDENT", "0")
    run()
    tw.release_cached_memory()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    want = run()
    need = before - torch.cuda.mem_get_info()[0]   # (the pool keeps it)
    tw.release_cached_memory()
    assert need > 100 << 20
    monkeypatch.delenv("TW_RESIDENT")
    held = torch.empty(torch.cuda.mem_get_info()[0] - need - (24 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = run()
    finally:
        del held
        torch.cuda.empty_cache()
        tw.release_cached_memory()
    assert np.abs(got).max() > 0 and np.array_equal(got, want)
