"""Large initial fields (above the pinned-staging size) whose very last row is not uniform: the
copy of the rows ends with the array."""
import re

import numpy as np
import pytest

import clip_b200 as cb
from test_gpu_two_pass import _config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(2048, 2047), (170, 161, 158)])
def test_a_field_without_uniform_rows(tmp_path, n):
    with cb.Solver(_config(tmp_path / "config.txt", n, "ppp"[: len(n)]), "fp64") as s:
        c = np.random.default_rng(5).random(s.extent)
        s.device_initializer(c)
        inner = tuple(slice(1, e - 1) for e in s.extent[: len(n)])
        assert np.array_equal(s.field("c").reshape(s.extent)[inner], c[inner])


def test_a_drop_at_the_last_row(tmp_path):
    path = tmp_path / "config.txt"
    _config(path, (2048, 2047), "pw")
    path.write_text(re.sub(r"center = .*", "center = [1000.5, 2046.5, 0.0]", path.read_text()))
    out = []
    for on_device in (False, True):
        with cb.Solver(str(path), "fp64") as s:
            s.init(on_device=on_device)
            out.append(s.interior_field("c"))
    # the device's tanh differs by a few units in the last place (test_gpu_init_device)
    assert np.abs(out[0] - out[1]).max() <= 8 * 2.3e-16
    assert out[0].max() > 0.9
