"""The two-pass 3D step (launch variant 7, the default of the FP32/FP16 paths) against the
one-pass march: every node's arithmetic is the same, so the state must be identical, at sizes
around its 32 x 4 tiles and for every kind of side, in which the boundary work differs."""
import numpy as np
import pytest

import clip_b200 as cb

pytestmark = pytest.mark.gpu

TYPES = {"p": ("periodic", "periodic"), "w": ("wall", "wall"), "s": ("slipwall", "wall"),
         "v": ("periodic", "periodic")}


def _config(path, n, sides):
    lines = ["case = drop", "finalStep = 10", f"N = [{n[0] + 2}, {n[1] + 2}, {n[2] + 2}]", "referenceLength = 6",
             "We = 8", "Re = 40", "gravity = [0, -1e-06, 0]", "mobility = 0.02", "interfaceWidth = 4", "muRatio = 10",
             "rhoRatio = 100", "geometry = [", "  {", '    type = "sphere"',
             f"    center = [{n[0] / 2 + 0.9}, {n[1] / 2 + 0.7}, {n[2] / 2 + 0.4}]", "    radius = 3", "    id = 0", "  }", "]",
             "boundary = ["]
    types = {"open": ["periodic", "periodic", "freeconvect", "velocity", "periodic", "periodic"],
             "inlet": ["periodic", "periodic", "wall", "velocity", "wall", "wall"]}.get(sides)
    if types is None:
        types = [t for s in sides for t in TYPES[s]]
    for side, t in zip(("x-", "x+", "y-", "y+", "z-", "z+"), types):
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


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
@pytest.mark.parametrize("n,sides", [((2, 2, 2), "ppp"), ((3, 5, 2), "ppp"), ((31, 4, 3), "pwp"), ((32, 8, 5), "pww"),
                                     ((33, 9, 4), "wpp"), ((34, 3, 6), "www"), ((65, 7, 7), "ppp"), ((64, 13, 9), "spw"),
                                     ((35, 11, 6), "inlet"), ((33, 10, 8), "open")])
def test_two_pass_equals_the_march(tmp_path, prec, n, sides):
    path = _config(tmp_path / "config.txt", n, sides)
    # 19 steps: one 16-step graph and single launches
    want, sums = _run(path, prec, 8, 19, sides != "open")
    for variant in (7, None):
        got, s2 = _run(path, prec, variant, 19, sides != "open")
        for f in want:
            assert np.isfinite(got[f]).all()
            assert np.array_equal(got[f], want[f]), f
        assert s2 == sums
