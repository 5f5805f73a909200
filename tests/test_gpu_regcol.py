"""The register-resident column passes against the generic kernels: every
line length, tiles that end inside the grid (nx not a multiple of the tile
width), both tile forms of the z pass, lines that are only along y or only
along z of that kind (the other axis generic), with and without SO coupling.

Bounds: both sides are the same split steps, so they differ by the rounding
of a few transforms per step (about 30 operations deep): 1e-12 of the largest
value in FP64, 1e-5 in FP32 (eps 6e-8 x sqrt of depth x 3 steps, doubled)."""
import numpy as np
import pytest

from tests.helpers import rel_err

pytestmark = pytest.mark.gpu

GRIDS = [(10, 128), (36, 192), (50, 256), (18, 384), (30, 512),          # q2D
         (10, 128, 16), (12, 192, 10), (18, 256, 8), (8, 384, 8), (10, 512, 8),       # y only
         (10, 16, 128), (12, 10, 192), (18, 8, 256), (10, 8, 384), (8, 8, 512),       # z only, small tiles
         (36, 60, 128), (50, 60, 192), (54, 60, 256), (36, 60, 384), (20, 60, 512),   # z, big tiles
         (20, 128, 256), (12, 256, 128)]                                              # both


@pytest.mark.parametrize("spin,precision,imag", [(1, "fp64", 1), (1, "fp32", 0), (2, "fp64", 0), (2, "fp32", 1)])
@pytest.mark.parametrize("n", GRIDS, ids=lambda n: "x".join(map(str, n)))
def test_matches_generic_kernels(n, spin, precision, imag):
    import fortress_b200 as F
    dim = len(n)
    gamma = (0.0,) * dim if n[-1] == 192 else (0.5, 0.3, 0.4)[:dim]
    p = dict(dim=dim, spin=spin, n=n, d=(0.3, 0.25, 0.2)[:dim], dt=1e-3 if imag else 5e-4, imag_time=imag,
             tau=(200.0, -5.0, 0.0) if spin == 1 else (300.0, 10.0, -8.0), gamma=gamma, alpha=(1.0, 1.3, 1.7),
             precision=precision, mag=0.1)
    rng = np.random.default_rng(5)
    ax = [np.linspace(-2, 2, m).reshape([-1 if q == a else 1 for q in range(dim)]) for a, m in enumerate(n)]
    g = np.exp(-sum(x * x for x in ax))
    shape = g.shape + (1,) * (3 - dim) + (2 * spin + 1,)
    phi = g.reshape(g.shape + (1,) * (4 - dim)) * (1 + 0.2 * rng.standard_normal(shape)) * np.exp(1j * rng.uniform(-1, 1, shape))
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
