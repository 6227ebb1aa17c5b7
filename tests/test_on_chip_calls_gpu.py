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
