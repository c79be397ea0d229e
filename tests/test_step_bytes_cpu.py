"""The byte model behind the bench's roofline counts what a step moves."""

import pytest

from meshtryoshka_gb300 import pipeline

SIZES = dict(G=1000, Nv=700, V=4000, F=7000, C=16, S=8, B=4, P=640_000, K=6000, T=100)


def test_only_marked_vertices_have_colours():
    every = pipeline.step_bytes(SIZES)
    some = pipeline.step_bytes({**SIZES, "seen": 1000})
    assert every["seen_marks"] == 0 and some["seen_marks"] > SIZES["V"]
    v = SIZES["V"]
    assert some["grid_sh_colors"] == every["grid_sh_colors"] // 4 + v  # a quarter of them, and the marks
    assert some["grid_sh_bwd"] < every["grid_sh_bwd"]


@pytest.mark.parametrize("touching", [0, 10, 6000])
def test_only_touching_faces_have_records(touching):
    found = pipeline.step_bytes({**SIZES, "touching": touching})["keys"]
    assert found == SIZES["B"] * SIZES["F"] * 48 + 44 * touching + 12 * SIZES["K"]
    assert found <= pipeline.step_bytes(SIZES)["keys"]
