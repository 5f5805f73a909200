"""Grouped and persistent batch passes at every size-specialised length on
both axes, both spins and precisions, against each instance stepped alone.
The passes differ in radix plans and in the order of the NORMC sums, so the
states agree to rounding: 6 steps of 4 transforms of up to 9 rounding stages
each are 216 roundings that add like a random walk, 15 units of rounding, and
the largest of a million values lies within 5 deviations: 75 units of 2^-24
(4.5e-6) or 2^-53 (8.3e-15; 1e-13 leaves room for the operators)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SHAPES = [(128, 192), (192, 256), (256, 384), (384, 512), (512, 128)]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mode", ["grouped", 0, 1, 2, 3, 4])
def test_batch_passes_at_every_length(mode, precision):
    import fortress_b200 as F
    from fortress_b200.batch import Batch
    insts = [dict(dim=2, spin=spin, n=n, d=(0.1, 0.12), dt=2e-4, imag_time=spin == 1, tau=(40.0, -3.0, 2.0),
                  gamma=(0.5, 0.3), alpha=(1.0, 1.2, 1.0), precision=precision)
             for n in SHAPES for spin in (1, 2)]
    singles, b = [F.Propagator(**p) for p in insts], Batch(insts)
    for k, p in enumerate(insts):
        rng = np.random.default_rng(50 + k)
        nx, ny = p["n"]
        x, y = np.linspace(-2, 2, nx), np.linspace(-2, 2, ny)
        g = np.exp(-x[:, None] ** 2 - y[None, :] ** 2)
        phi = rng.uniform(0.5, 1.0, (nx, ny, 1, 2 * p["spin"] + 1)) * g[:, :, None, None] * np.exp(0.3j)
        phi /= np.sqrt(0.1 * 0.12 * (np.abs(phi) ** 2).sum())
        for q in (singles[k], b[k]):
            q.set_state(phi)
            if p["imag_time"]:
                q.normt()
    if mode == "grouped":
        b.mode(grouped=True)
    else:
        b.mode(persistent=True)
        assert b.variant(mode) == mode
    b.config(width=4, steps_per_graph=4)
    b.step(6)
    tol = 1e-13 if precision == "fp64" else 4.5e-6
    for k, s in enumerate(singles):
        s.step(6)
        sa, sb = np.asarray(b[k].state()), np.asarray(s.state())
        assert np.abs(sa - sb).max() <= tol * np.abs(sb).max(), (insts[k]["n"], insts[k]["spin"])
        assert np.allclose(b[k].normc(), s.normc(), rtol=10 * tol, atol=0)
