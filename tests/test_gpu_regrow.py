"""The register-resident spin-1 row pass (AUTO on grids of many rows) against
the block pass: every line length, row counts that leave warps with a partial
last batch, both time directions, with and without SO coupling, and the
real-space snapshots behind CONV.

Bounds: the passes differ by the rounding of two transforms and one
real-space update per step: 1e-12 of the largest value in FP64, 1e-5 in FP32
(eps 6e-8 x sqrt of the depth x 3 steps, doubled); CONV is a difference of
successive states, so it carries the same absolute error."""
import numpy as np
import pytest

from tests.helpers import rel_err

pytestmark = pytest.mark.gpu

GRIDS = [(128, 30, 72), (192, 30, 72), (256, 64, 32), (256, 30, 72), (384, 30, 72), (512, 32, 64), (128, 50, 60)]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("imag", [1, 0])
@pytest.mark.parametrize("n", GRIDS, ids=lambda n: "x".join(map(str, n)))
def test_matches_block_pass(n, imag, precision):
    import fortress_b200 as F
    gamma = (0.0, 0.0, 0.0) if n[1] == 50 else (0.5, 0.3, 0.4)
    p = dict(dim=3, spin=1, n=n, d=(0.1, 0.25, 0.2), dt=1e-3 if imag else 5e-4, imag_time=imag, tau=(400.0, -15.0, 0.0),
             gamma=gamma, alpha=(1.0, 1.3, 1.7), precision=precision, mag=0.1)
    rng = np.random.default_rng(6)
    ax = [np.linspace(-2, 2, m).reshape([-1 if q == a else 1 for q in range(3)]) for a, m in enumerate(n)]
    g = np.exp(-sum(x * x for x in ax))[..., None]
    shape = n + (3,)
    phi = g * (1 + 0.2 * rng.standard_normal(shape)) * np.exp(1j * rng.uniform(-1, 1, shape))
    got = []
    for kernels in ("auto", "block-row"):
        q = F.Propagator(**p, kernels=kernels)
        q.set_state(phi)
        q.normt()
        q.step(3)
        got.append((q.state(), q.normc(), q.conv()))
        q.close()
    tol = 1e-12 if precision == "fp64" else 1e-5
    assert rel_err(got[0][0], got[1][0]) < tol
    assert np.allclose(got[0][1], got[1][1], rtol=tol, atol=0)
    assert abs(got[0][2] - got[1][2]) <= 2 * tol * np.abs(got[1][0]).max()
