"""Field readback: values converted on the GPU, rows staged in bounded pieces, results of any row
stride. What is written comes back exactly (FP32 and FP64 values; 16-bit storage: the rounded value, or the
sum hi + lo of the pair), and nothing between the rows of a strided result is touched."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Mx,My", [(8, 4), (40, 33), (300, 1025), (2100, 4100)])   # the last: more than one piece
@pytest.mark.parametrize("prec,cpst", [("f32", "00"), ("f64", "00"), ("bf16", "00"), ("fp16", "split")])
def test_written_fields_read_back(tw, Mx, My, prec, cpst):
    rng = np.random.default_rng(Mx + My)
    s = tw.Solver(Mx, My, 1, max(Mx, My), 1e-4, precision=prec, cpst=cpst, max_steps=1)
    for g, f in ((tw.NN, 0), (tw.MN, 0), (tw.NM, 0), (tw.MM, 1)):
        a = rng.standard_normal(s.shape(g)).astype(np.float32).astype(np.float64)
        s.write_field(g, f, a)
        got = s.read_field(g, f)
        if prec == "bf16":
            u = a.astype(np.float32).view(np.uint32).astype(np.uint64)
            want = (((u + 0x7FFF + ((u >> 16) & 1)) >> 16) << 16).astype(np.uint32).view(np.float32).astype(np.float64)
        elif prec == "fp16":
            h = a.astype(np.float16).astype(np.float32)
            lo = (a.astype(np.float32) - h).astype(np.float16).astype(np.float32)
            want = (h + lo).astype(np.float64)
        else:
            want = a
        assert np.array_equal(got, want), (g, f)
        r, c = got.shape
        wide = np.full((r, c + 5), -7.0)
        rc = tw.lib().tw_read_field(s.h, g, f, wide.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), c + 5)
        assert rc == 0 and np.array_equal(wide[:, :c], want) and (wide[:, c:] == -7.0).all()
    s.close()
