"""Edge strips of the per-warp kernel (the columns at the periodic seam): one value a row across the seam
is staged with the others and 16-bit pairs travel as the words that hold them. Widths put the seam at each
place in a strip (first and last lane pair, odd and even columns, the last strip one column wide); all
results bit-identical to the oracle's. TMA handles run the same strips as work items of 6 rows and
take their own items in alternating order."""
import numpy as np
import pytest

from cases import elastic_case, product_elastic
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

FORMS = [("f32", "00"), ("f32", "6C"), ("f32", "3R"), ("f64", "00"), ("fp16", "split"), ("bf16", "split"), ("bf16", "00")]


@pytest.mark.parametrize("My", [54, 55, 56, 57, 111, 112, 113])
@pytest.mark.parametrize("precision,cpst", FORMS)
def test_edge_strips_bit_identical(monkeypatch, My, precision, cpst):
    monkeypatch.setenv("TW_RESIDENT", "0")   # (such grids would run on chip)
    case = elastic_case(60, My, seed=My, cpst=cpst, Nt=25, model="random")
    want = orc.elastic_run(case, precision)
    got = product_elastic(case, precision)
    for k, v in got["fields"].items():
        assert np.array_equal(v, want.fields[k]), k
    assert np.array_equal(got["traces"], want.traces)


@pytest.mark.parametrize("energy", [False, True])
@pytest.mark.parametrize("My", [180, 236, 237, 299, 301])
def test_strip_items_of_the_tma_step(monkeypatch, My, energy):
    monkeypatch.setenv("TW_RESIDENT", "0")
    case = elastic_case(75, My, seed=My, cpst="00", Nt=25, model="random")
    want = orc.elastic_run(case, "f32")
    got = product_elastic(case, "f32", energy=energy)
    for k, v in got["fields"].items():
        assert np.array_equal(v, want.fields[k]), k
    assert np.array_equal(got["traces"], want.traces)
