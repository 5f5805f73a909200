"""The unfused FFT and BFT on lengths with and without a compiled kernel
(each axis takes the register-resident single transforms or the generic pass
by its own length) against torch's FFT in FP64, both precisions and spins, and
after a change of the kernel family, which changes the passes.

Bound: a transform of N values rounds like sqrt(log2 N) to log2 N operations
in a row; 2 log2 N units of rounding of the largest value."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

GRIDS = [(20, 128), (128, 60), (192, 192), (10, 256), (36, 384), (16, 512), (24, 128, 192), (16, 256, 30), (18, 20, 384),
         (10, 512, 128), (128, 384, 256), (20, 12, 30)]


@pytest.mark.parametrize("spin,precision", [(1, "fp64"), (1, "fp32"), (2, "fp64"), (2, "fp32")])
@pytest.mark.parametrize("n", GRIDS, ids=lambda n: "x".join(map(str, n)))
def test_fft_and_bft(n, spin, precision):
    import fortress_b200 as F
    dim, shape = len(n), tuple(n) + (1,) * (3 - len(n)) + (2 * spin + 1,)
    rng = np.random.default_rng(sum(n))
    phi = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    unit = 2.0 ** -53 if precision == "fp64" else 2.0 ** -24
    tol = 2 * math.log2(np.prod(n)) * unit
    want = torch.fft.fftn(torch.from_numpy(phi).cuda(), dim=tuple(range(dim))).cpu().numpy()
    q = F.Propagator(dim=dim, spin=spin, n=n, d=(0.1,) * dim, dt=1e-3, imag_time=True, tau=(1.0, 0.1, 0.1),
                     gamma=(0.5, 0.3, 0.4)[:dim], alpha=(1.0, 1.0, 1.0), precision=precision)
    for kernels in ("auto", "fast-row", "auto"):
        q.set_kernels(kernels)
        q.set_state(phi)
        q.FFT()
        got = np.asarray(q.state()).reshape(shape)
        assert np.abs(got - want).max() <= tol * np.abs(want).max(), kernels
        q.BFT()
        back = np.asarray(q.state()).reshape(shape)
        assert np.abs(back - phi).max() <= 2 * tol * np.abs(phi).max(), kernels
    q.close()
