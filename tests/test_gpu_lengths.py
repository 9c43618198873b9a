"""Every line length that the Green's function passes are instantiated for,
against the FP32 oracle: whole-box operators (all planes in and out) and one
time step (the pruned x3 transform), on boxes whose column pairs and rows do
not fill the last block.

Tolerance: relative L2 <= 1e-5, the bound of the operators and of a step
elsewhere in these tests.
"""
import ctypes as C

import numpy as np
import pytest

from relax_b200 import _lib
from relax_b200.api import Relax
from relax_b200.config import Event, Fault, Simulation

from cases import rel_l2, tensor_array

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

X3 = (24, 32, 36, 48, 54, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256, 288, 384, 512)
X2 = (24, 27, 32, 36, 48, 54, 64, 72, 81, 96, 108, 128, 144, 162, 192, 216, 243, 256, 288, 324, 384, 432, 486, 512)
X1 = (24, 32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 216, 256, 288, 324, 384, 432, 512)


def green_error(oracle, sx1, sx2, sx3, gam=8.3e-4):
    rng = np.random.default_rng(sx1 + 1000 * sx2 + 7 * sx3)
    dx = (0.5, 0.4, 0.25)
    c = np.zeros((3, sx3, sx2, sx1 + 2), np.float32)
    c[..., :sx1] = rng.standard_normal((3, sx3, sx2, sx1))
    t = np.zeros((3, sx2, sx1 + 2), np.float32)
    t[..., :sx1] = 0.1 * rng.standard_normal((3, sx2, sx1))
    dc, dt = [torch.from_numpy(v).cuda() for v in c], [torch.from_numpy(v).cuda() for v in t]
    cr, tr = c.copy(), t.copy()
    oracle.green(cr, tr, sx1, sx2, sx3, dx, 1.0, 1.0, gam)
    _lib.check(_lib.load().relax_op_green(*[C.c_void_p(v.data_ptr()) for v in dc + dt], sx1, sx2, sx3, *dx, 1.0, 1.0,
                                          gam, None))
    torch.cuda.synchronize()
    return rel_l2(np.stack([v.cpu().numpy() for v in dc])[..., :sx1], cr[..., :sx1])


def step_errors(oracle, sx1, sx2, sx3):
    lid = (sx3 // 6) * 1.0
    sim = Simulation(sx1=sx1, sx2=sx2, sx3=sx3, dx1=1.0, dx2=1.0, dx3=1.0, beta=0.2, nyquist=2.0, lambda_=1.0, mu=1.0,
                     gam=8.3e-4, interval=1.0e6, odt=-1, tscale=1.0, nonlinear=[(lid, 1.0, 3.0, 0.0)],
                     events=[Event(0.0, [Fault(1.0, -3.0, 0.0, 0.5, 6.0, 4.0, 30.0, 60.0, 45.0)])])
    with Relax(sim) as r:
        r.coseismic()
        log = r.step()
        got = {k: r.field(k) for k in ("u", "tau", "gamma")}
    _, ref = oracle.run(sim, 1, dt_schedule=[log[1]])
    return {"u": rel_l2(got["u"][..., :-2], ref["u"][..., :-2]),
            "tau": rel_l2(tensor_array(got["tau"]), tensor_array(ref["tau"]))}


@pytest.mark.parametrize("sx3", X3)
def test_x3_lengths(oracle32, sx3):
    assert green_error(oracle32, 24, 27, sx3) < 1e-5     # odd sx2: the wavenumbers are not symmetric
    errs = step_errors(oracle32, 24, 18, sx3)
    assert max(errs.values()) < 1e-5, errs


@pytest.mark.parametrize("sx2", X2)
def test_x2_lengths(oracle32, sx2):
    assert green_error(oracle32, 24, sx2, 32) < 1e-5


@pytest.mark.parametrize("sx1", X1)
def test_x1_lengths(oracle32, sx1):
    assert green_error(oracle32, sx1, 18, 24) < 1e-5
    errs = step_errors(oracle32, sx1, 27, 24)            # odd sx2: the last row of a plane has no partner
    assert max(errs.values()) < 1e-5, errs
