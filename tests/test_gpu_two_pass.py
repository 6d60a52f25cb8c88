"""The two-pass step (the default launch: variant 7 of the 3D FP32/FP16 paths, 4 of the 3D FP64
path, 3 of the 2D paths) against the one-pass march: every node's arithmetic is the same, so the
state must be identical, at sizes around its 32 x 4 tiles and for every kind of side, in which
the boundary work differs."""
import numpy as np
import pytest

import clip_b200 as cb

pytestmark = pytest.mark.gpu

TYPES = {"p": ("periodic", "periodic"), "w": ("wall", "wall"), "s": ("slipwall", "wall"),
         "v": ("periodic", "periodic")}


def _config(path, n, sides):
    dim = len(n)
    size = [v + 2 for v in n] if dim == 3 else [n[0], n[1], 1]
    center = [n[a] / 2 + 0.9 - 0.2 * a for a in range(dim)] + [0.0] * (3 - dim)
    lines = ["case = drop", "finalStep = 10", f"N = {size}", "referenceLength = 6",
             "We = 8", "Re = 40", "gravity = [0, -1e-06, 0]", "mobility = 0.02", "interfaceWidth = 4", "muRatio = 10",
             "rhoRatio = 100", "geometry = [", "  {",
             f'    type = "{"sphere" if dim == 3 else "circle"}"', f"    center = {center}", "    radius = 3", "    id = 0", "  }", "]",
             "boundary = ["]
    types = {"open": ["periodic", "periodic", "freeconvect", "velocity", "periodic", "periodic"],
             "inlet": ["periodic", "periodic", "wall", "velocity", "wall", "wall"]}.get(sides)
    if types is None:
        types = [t for s in sides for t in TYPES[s]]
    for side, t in zip(("x-", "x+", "y-", "y+", "z-", "z+")[: 2 * dim], types):
        lines += ["  {", f'    side = "{side}"', f'    type = "{t}"']
        lines += ["    value = [0, -0.01, 0]"] if t == "velocity" else []
        lines += ["  },"]
    path.write_text("\n".join(lines + ["]", ""]))
    return str(path)


def _run(path, prec, variant, steps, monitored):
    with cb.Solver(path, prec) as s:
        if variant is not None:
            s.set_launch(variant, 3)
        s.init()
        s.solve(steps)
        sums = s.solve_monitored(1) if monitored else None
        return {f: s.interior_field(f) for f in ("c", "vel", "f_post", "g_post")}, sums


def _compare(path, prec, march, two_pass, monitored):
    # 19 steps: one 16-step graph and single launches
    want, sums = _run(path, prec, march, 19, monitored)
    for variant in (two_pass, None):
        got, s2 = _run(path, prec, variant, 19, monitored)
        for f in want:
            assert np.isfinite(got[f]).all()
            assert np.array_equal(got[f], want[f]), f
        assert s2 == sums


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("n,sides", [((2, 2, 2), "ppp"), ((3, 5, 2), "ppp"), ((31, 4, 3), "pwp"), ((32, 8, 5), "pww"),
                                     ((33, 9, 4), "wpp"), ((34, 3, 6), "www"), ((65, 7, 7), "ppp"), ((64, 13, 9), "spw"),
                                     ((35, 11, 6), "inlet"), ((33, 10, 8), "open")])
def test_two_pass_equals_the_march_3d(tmp_path, prec, n, sides):
    path = _config(tmp_path / "config.txt", n, sides)
    _compare(path, prec, 2 if prec == "fp64" else 8, 4 if prec == "fp64" else 7, sides != "open")


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("n,sides", [((2, 2), "pp"), ((3, 5), "pw"), ((31, 4), "wp"), ((32, 8), "ww"), ((33, 9), "pp"),
                                     ((64, 3), "sp"), ((65, 13), "pw"), ((35, 11), "inlet"), ((33, 10), "open")])
def test_two_pass_equals_the_march_2d(tmp_path, prec, n, sides):
    _compare(_config(tmp_path / "config.txt", n, sides), prec, 0, 3, False)


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
@pytest.mark.parametrize("rows", [1, 5, 16, 64])
def test_two_pass_batch_equals_the_march(prec, rows):
    """Rows per work item that the 4-row tiles do not divide, and items longer than a case."""
    texts = [cb.seeded_case_config(31, i) for i in range(5)]
    out = []
    for variant, seg in ((1, 8), (3, rows)):
        with cb.Batch(texts, prec, texts=True) as b:
            b.set_launch(variant, seg)
            b.init()
            b.solve(19)
            out.append([b.case(i).interior_field(f) for i in range(5) for f in ("c", "vel", "g")])
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_two_pass_work_array_is_optional(tmp_path, prec):
    """A solver whose state fits but not the work array is created all the same, and marches."""
    import torch

    path = _config(tmp_path / "config.txt", (8192, 1024), "pw")
    with cb.Solver(path, prec) as s:
        need = s.info().device_bytes
        s.set_launch(0, 0)
        s.init()
        s.solve(3)
        want = s.interior_field("f_post")
        s.set_launch(3, 0)  # loads its kernels too
        s.solve(1)
    work = 8192 * 1024 * 8  # at least; allocations round up to 2 MB
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (need - work // 4), dtype=torch.uint8, device="cuda")
    s = cb.Solver(path, prec)
    del filler
    torch.cuda.empty_cache()
    try:
        assert s.info().device_bytes <= need - work
        s.init()
        s.solve(3)
        assert np.array_equal(s.interior_field("f_post"), want)
    finally:
        s.close()
