"""The END stress pass with bulk copies (boxes of at least 592 tiles of 1024
points): a box whose last tile is partly empty against the FP32 oracle (the
bound of one step, relative L2 <= 1e-5), and two contexts of one deck bit for
bit over many steps (a copy that overtook a read would differ)."""
import numpy as np
import pytest

from relax_b200.api import Relax
from relax_b200.config import linear_maxwell, powerlaw_thrust

from test_gpu_lengths import step_errors

pytestmark = pytest.mark.gpu


def test_partly_empty_tile(oracle32):
    errs = step_errors(oracle32, 108, 108, 108)          # 615.09 tiles
    assert max(errs.values()) < 1e-5, errs


@pytest.mark.parametrize("sim", [linear_maxwell(128, 128), powerlaw_thrust(256, 128)], ids=["128^3", "256^2x128"])
def test_contexts_agree_bit_for_bit(sim):
    sim.interval = 1.0e6
    got = []
    for _ in range(2):
        with Relax(sim) as r:
            r.coseismic()
            logs = [r.step() for _ in range(40)]
            got.append((logs, r.field("u"), r.field("tau"), r.field("gamma")))
    assert got[0][0] == got[1][0]
    for a, b in zip(got[0][1:], got[1][1:]):
        assert np.array_equal(a, b)
