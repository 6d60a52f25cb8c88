"""The two-pass step's work array gives way: what a solver or batch allocates after it still
fits where the memory without that array suffices, and the steps then march, with the same
bits.  Each test leaves less free memory than the allocation wants, but more than it wants
beyond the array."""
import contextlib

import numpy as np
import pytest

import clip_b200 as cb
from test_gpu_two_pass import _config

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    import torch

    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@contextlib.contextmanager
def _full_but(leave):
    """All free device memory but `leave` bytes is taken."""
    import torch

    hold = [torch.empty(_free() - leave, dtype=torch.uint8, device="cuda")]
    try:
        yield
    finally:
        hold.clear()
        torch.cuda.empty_cache()


def _padded(n):
    """Nodes of the padded layout (rows start at 31, row lengths are multiples of 32)."""
    return (31 + n[0] + 2 + 31) // 32 * 32 * (n[1] + 2) * (n[2] + 2 if len(n) == 3 else 1)


TARGET = np.array([500.0, 500.0])
# call: precision, grid, the call, and the bytes it allocates (None: as measured, for what it keeps)
CALLS = {
    "field": ("fp32", (2048, 2048), lambda s, tmp: s.field("c"), None),
    "vts": ("fp32", (2048, 2048), lambda s, tmp: s.write_vts(tmp, "a", "binary32"), None),
    "monitored": ("fp16", (4, 640, 640), lambda s, tmp: s.solve_monitored(1), None),
    "adjoint": ("fp64", (1024, 1024), lambda s, tmp: s.adjoint(2, TARGET, None, 2), None),
    "tangent": ("fp64", (1024, 1024), lambda s, tmp: s.tangent(2, TARGET, dparams=[0.0, 1.0, 0.0]),
                16 * 41 * _padded((1024, 1024))),
}


@pytest.mark.parametrize("call", list(CALLS))
def test_a_solvers_later_allocations_fit(tmp_path, call):
    prec, n, do, need = CALLS[call]
    path = _config(tmp_path / "config.txt", n, "pww"[: len(n)])
    with cb.Solver(path, prec) as s:  # with all memory: the bytes, and the state afterwards
        two_pass = s.get_launch()[0]
        s.init()
        s.solve(2)
        before = _free()
        do(s, tmp_path)
        need = need or before - _free()
        s.solve(3)
        want = s.interior_field("c")
    with cb.Solver(path, prec) as s:
        assert s.get_launch()[0] == two_pass
        s.init()
        s.solve(2)
        with _full_but(need - min(need, 8 * _padded(n)) // 2):
            do(s, tmp_path)
        assert s.get_launch()[0] == 0
        s.solve(3)
        assert np.array_equal(s.interior_field("c"), want)
        s.set_launch(two_pass, 4)  # accepted as before; marches
        assert s.get_launch()[:2] == (0, 4)


def test_a_read_after_a_read_that_did_not_fit(tmp_path):
    """The larger read frees the stage before it asks for its own; the next one needs a stage too."""
    with cb.Solver(_config(tmp_path / "config.txt", (2048, 2048), "pw"), "fp32") as s:
        s.init()
        s.solve(2)
        want = s.field("c")
        with _full_but(4 * MB):
            with pytest.raises(cb.ClipError, match="out of memory"):
                s.field("g_post")
            assert np.array_equal(s.field("c"), want)


def _batch(tmp_path, prec):
    paths = [_config(tmp_path / f"config{i}.txt", (1024, 1024 + 32 * i), "pw") for i in range(4)]
    return cb.Batch([open(p).read() for p in paths], prec, texts=True)


def _states(b):
    return [b.case(i).interior_field(f) for i in range(4) for f in ("c", "vel")]


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_a_batch_fits_without_the_work_arrays(tmp_path, prec):
    before = _free()
    with _batch(tmp_path, prec) as b:
        used = before - _free()
        b.init()
        b.solve(19)
        want = _states(b)
    with _full_but(used - 2 * 8 * _padded((1024, 1024))):
        b = _batch(tmp_path, prec)
    with b:
        assert b.get_launch()[0] == 0
        b.set_launch(3, 8)
        b.init()
        b.solve(19)
        for x, y in zip(_states(b), want):
            assert np.array_equal(x, y)


def test_a_batch_gives_way_to_a_field_read(tmp_path):
    with _batch(tmp_path, "fp32") as b:
        b.init()
        b.solve(17)
        b.solve(20)
        want = _states(b)
    with _batch(tmp_path, "fp32") as b:
        b.init()
        b.solve(17)
        with _full_but(4 * MB):  # the field of a case takes 8 MB
            c = b.case(2).interior_field("c")
        assert np.isfinite(c).all() and b.get_launch()[0] == 0
        b.solve(20)
        for x, y in zip(_states(b), want):
            assert np.array_equal(x, y)
