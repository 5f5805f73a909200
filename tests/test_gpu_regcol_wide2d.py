"""The q2D column pass of spin-2 lines of 192 and 256 points on grids wide
enough for its second tile form (more than two x positions per SM), against
the generic kernels: at the first width past the line, a width that the
four-position tiles do not divide, and the largest compiled row length.

Bounds as in test_gpu_regcol.py: the rounding of a few transforms per step,
1e-12 of the largest value in FP64, 1e-5 in FP32."""
import numpy as np
import pytest

from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,imag", [("fp64", 1), ("fp64", 0), ("fp32", 1), ("fp32", 0)])
@pytest.mark.parametrize("n", [(300, 192), (450, 192), (512, 192), (300, 256), (450, 256), (512, 256)],
                         ids=lambda n: "x".join(map(str, n)))
def test_matches_generic_kernels(n, precision, imag):
    import fortress_b200 as F
    p = dict(dim=2, spin=2, n=n, d=(0.1, 0.12), dt=1e-3 if imag else 5e-4, imag_time=imag, tau=(300.0, 10.0, -8.0),
             gamma=(0.0, 0.0) if n[0] == 300 else (0.5, 0.3), alpha=(1.0, 1.3, 1.7), precision=precision, mag=0.1)
    rng = np.random.default_rng(7)
    x, y = np.linspace(-2, 2, n[0]), np.linspace(-2, 2, n[1])
    g = np.exp(-x[:, None] ** 2 - y[None, :] ** 2)[:, :, None, None]
    shape = (n[0], n[1], 1, 5)
    phi = g * (1 + 0.2 * rng.standard_normal(shape)) * np.exp(1j * rng.uniform(-1, 1, shape))
    got = []
    for kernels in ("auto", "generic"):
        q = F.Propagator(**p, kernels=kernels)
        q.set_state(phi)
        q.normt()
        q.step(3)
        got.append((q.state(), q.normc()))
        q.close()
    tol = 1e-12 if precision == "fp64" else 1e-5
    assert rel_err(got[0][0], got[1][0]) < tol
    assert np.allclose(got[0][1], got[1][1], rtol=tol, atol=0)
