"""The adjoint's vector path (points away from the closures, the penalties and the seam) beside its
general one, at sizes where the vectors begin, end and leave columns over.

FP64: the dot-product identity of the state map to 1e-12 (it holds only if every point's transposed
operators are exact). FP32: the same identity to 2e-5 (30 steps of FP32 sums: some 1e-6), and gradients
against the FP64 ones to 1e-4 in the 2-norm (the state they come from carries 1e-6 to 1e-5).
Segments recomputed on chip and by single steps give the same gradient bit for bit.
"""
import numpy as np
import pytest

from cases import elastic_case, load_twave
from test_adjoint_gpu import random_state, rcvs_for, single_field_mask, solver

pytestmark = pytest.mark.gpu
KEYS = ("NN", "MN", "NM", "MM0", "MM1")
SIZES = [(13, 14), (14, 16), (20, 17), (33, 34), (21, 35), (40, 61), (27, 130)]


def _run(case, prec, x, y, nt, K):
    tw = load_twave()
    out = []
    for adjoint in (False, True):
        s = solver(tw, case, precision=prec, source=False)
        for (g, f), a in zip([(tw.NN, 0), (tw.MN, 0), (tw.NM, 0), (tw.MM, 0), (tw.MM, 1)], x):
            s.write_field(g, f, a)
        if adjoint:   # residual trace - obs = y
            out.append(s.adjoint_gradient(nt, out[0] - y, ckpt_every=K, state=True))
        else:
            s.run(nt)
            out.append(s.read_receivers())
        s.close()
    return out


@pytest.mark.parametrize("prec,tol", [("f64", 1e-12), ("f32", 2e-5)])
@pytest.mark.parametrize("Mx,My", SIZES)
def test_dot_product_identity(Mx, My, prec, tol):
    tw = load_twave()
    nt, den = 30, max(Mx, My)
    case = elastic_case(Mx, My, seed=3, Nt=nt, den_dx=den, rcvs=rcvs_for(Mx, My, den))
    x = [np.float32(a).astype(np.float64) for a in random_state(case, 1)]
    y = np.random.default_rng(2).standard_normal((len(case.rcvs), 2, nt)) * single_field_mask(tw, case)
    d, g = _run(case, prec, x, y, nt, 7)
    lhs, rhs = float(np.sum(d * y)), float(sum(np.sum(a * g["state"][k]) for a, k in zip(x, KEYS)))
    assert abs(lhs - rhs) <= tol * max(abs(lhs), np.linalg.norm(d) * np.linalg.norm(y))


@pytest.mark.parametrize("Mx,My", [(20, 17), (40, 61), (130, 150)])
def test_fp32_gradient_against_fp64_and_single_steps(Mx, My, monkeypatch):
    tw = load_twave()
    nt, den = 30, max(Mx, My)
    case = elastic_case(Mx, My, seed=3, Nt=nt, den_dx=den, rcvs=rcvs_for(Mx, My, den))
    x = [np.float32(a).astype(np.float64) for a in random_state(case, 1)]
    y = np.random.default_rng(2).standard_normal((len(case.rcvs), 2, nt)) * single_field_mask(tw, case)
    _, g32 = _run(case, "f32", x, y, nt, 7)
    _, g64 = _run(case, "f64", x, y, nt, 7)
    monkeypatch.setenv("TW_RESIDENT", "0")
    _, one = _run(case, "f32", x, y, nt, 7)
    for k in g32["grid"]:
        assert np.linalg.norm(g32["grid"][k] - g64["grid"][k]) <= 1e-4 * np.linalg.norm(g64["grid"][k]), k
        assert np.array_equal(g32["grid"][k], one["grid"][k]), k
    for k in g32["state"]:
        assert np.array_equal(g32["state"][k], one["state"][k]), k
