"""The END stress pass with bulk copies on the transient (Burgers) rheology:
a box whose last tile is partly empty against the FP32 oracle (the bounds of
the transient runs: relative L2 <= 1e-5 after one step, 1e-4 after more), and
a batch of two members bit for bit against the members alone."""
import pytest

from cases import transient_small
from test_gpu_batch import _alone, _batched, _same, _variant
from test_gpu_step import check_logs, compare
from test_gpu_transient import _gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsteps", [1, 3])
def test_partly_empty_tile(oracle32, nsteps):
    sim = transient_small(linear=True, nonlinear=True, viscous=True, sx=108, sz=108)   # 615.09 tiles
    glogs, gtm, gf = _gpu(sim, nsteps)
    rlogs, rf = oracle32.run(sim, nsteps, dt_schedule=[l[1] for l in glogs[1:]])
    tol = 1e-5 if nsteps == 1 else 1e-4
    check_logs(glogs, rlogs, 10 * tol)
    for g, o in zip(gtm, rf["tm_transient"][1:]):
        for a, b in zip(g, o):
            assert abs(a - b) <= 1e-5 * abs(b), (g, o)
    compare(gf, rf, tol)


def test_batch_matches_members_alone():
    base = transient_small(linear=True, nonlinear=True, viscous=True, sx=108, sz=108)
    sims = [_variant(base, k) for k in range(2)]
    outs, _ = _batched(sims, 4)
    for k, s in enumerate(sims):
        _same(outs[k], _alone(s, 4))
