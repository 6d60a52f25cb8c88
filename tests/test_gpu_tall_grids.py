"""Grids of more rows or planes than a launch of the two-pass step covers (65,535 blocks of 4
rows, 65,535 planes), and the largest that it does: created, stepped and, where the march runs
instead, with the march's state.  The drop lies where the launch would end."""
import re

import numpy as np
import pytest

import clip_b200 as cb
from test_gpu_two_pass import _config

pytestmark = pytest.mark.gpu


def _tall(path, n, sides, axis, at):
    _config(path, n, sides)
    center = [n[a] / 2 + 0.5 if a < len(n) else 0.0 for a in range(3)]
    center[axis] = at + 0.4
    path.write_text(re.sub(r"center = .*", f"center = {center}", path.read_text()))
    return str(path)


def _run(path, prec, variant, fields, monitored):
    with cb.Solver(path, prec) as s:
        if variant is not None:
            s.set_launch(variant)
        s.init()
        s.solve(3)
        sums = s.solve_monitored(1) if monitored else s.monitors()
        return [s.interior_field(f) for f in fields], sums


def _same(path, prec, march, two_pass, fields, monitored):
    want, w = _run(path, prec, march, fields, monitored)
    for variant in (None, two_pass):
        got, g = _run(path, prec, variant, fields, monitored)
        for a, b in zip(want, got):
            assert np.isfinite(b).all() and np.array_equal(a, b)
        assert w == g


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("n,sides", [((2, 262138), "pp"), ((2, 262139), "pp"), ((2, 262200), "pw"), ((3, 524270), "wp")])
def test_rows_2d(tmp_path, prec, n, sides):
    path = _tall(tmp_path / "config.txt", n, sides, 1, 262140 if n[1] < 300000 else 524280 - 16)
    _same(path, prec, 0, 3, ("c", "vel", "f_post", "g_post"), False)


def test_rows_2d_open(tmp_path):
    path = _tall(tmp_path / "config.txt", (2, 262200), "open", 1, 262140)
    _same(path, "fp32", 0, 3, ("c", "vel", "f_post", "g_post"), False)


def test_rows_3d(tmp_path):
    path = _tall(tmp_path / "config.txt", (2, 262200, 2), "wpp", 1, 262140)
    _same(path, "fp16", 8, 7, ("c", "vel"), True)


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nz", [65533, 65534, 65600])
def test_planes(tmp_path, prec, nz):
    # fields of more than 65,535 planes cannot be read back: their sums are compared
    path = _tall(tmp_path / "config.txt", (2, 2, nz), "ppw", 2, min(nz - 2, 65536))
    _same(path, prec, 2 if prec == "fp64" else 8, 4 if prec == "fp64" else 7, ("c", "vel", "g") if nz <= 65533 else (), True)


@pytest.mark.parametrize("ny", [70000, 262200])
def test_autotune_skips_shapes_that_a_launch_cannot_cover(tmp_path, ny):
    """One row per block is such a shape on both grids."""
    with cb.Solver(_tall(tmp_path / "config.txt", (2, ny), "pw", 1, ny // 2), "fp32") as s:
        s.init()
        want = s.interior_field("c")
        variant, seg, ms = s.autotune(2)
        assert ms < 1e6 and (variant == 3 or seg > 1)
        assert s.steps == 0 and np.array_equal(s.interior_field("c"), want)
        s.solve(3)
        assert np.isfinite(s.interior_field("c")).all()
