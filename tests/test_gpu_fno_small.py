"""The smallest learned-guess problems: a batch of one.

A pair of products with one B for both and batch = 1 (include/fno.h allows it
where sAb == 0 and sBb != 0) is the two products one after the other, bit for
bit, and a network of one channel and one sample, whose spectral stages are
such pairs, runs forward and backward.  The FP32 GEMM path is the reference of
the network: both paths follow the FP64 oracle to the bounds of
test_gpu_fno.py, so they differ by at most the sum of those (outputs 1e-2 +
1e-4, gradients 5e-2 + 1e-3 of the largest entry)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("M,N,K,beta", [(1, 1, 1, 0.0), (16, 20, 128, 0.0), (33, 21, 70, 1.0), (130, 66, 9, 0.0)])
def test_pair_on_one_shared_operand(M, N, K, beta):
    from fortress_b200 import fno as FN
    L = FN.lib()
    gen = torch.Generator("cuda").manual_seed(M + N)
    A = [torch.randn(M * K, device="cuda", generator=gen) for _ in range(2)]
    B = torch.randn(K * N, device="cuda", generator=gen)
    C = [torch.randn(M * N, device="cuda", generator=gen) for _ in range(2)]
    want = [c.clone() for c in C]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    sA, sB, sC = (0, K, 1), (K * N, N, 1), (M * N, N, 1)
    for q in range(2):
        assert 0 == L.fno_gemm_tc(1, M, N, K, 0.5, _p(A[q]), 0, *sA, _p(B), *sB, beta, _p(want[q]), *sC, _p(err), st)
    assert 0 == L.fno_gemm_tc2(1, M, N, K, 0.5, _p(A[0]), _p(A[1]), *sA, _p(B), _p(B), *sB, beta, _p(C[0]), _p(C[1]), *sC,
                               _p(err), st)
    torch.cuda.synchronize()
    assert err.item() == 0
    assert torch.equal(C[0], want[0]) and torch.equal(C[1], want[1])


def test_network_of_one_channel_and_one_sample():
    from fortress_b200 import fno as FN
    cfg = dict(width=1, modes=4, layers=2, hidden=16)
    p = FN.init_params(cin=7, cout=6, seed=3, **cfg)
    a = FN.input_channels(np.random.default_rng(5).uniform(-1, 1, size=(1, 5)), 16)
    target = torch.randn(6, 256, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    out, grad = [], []
    for tc in (True, False):
        net = FN.FNO(16, 1, params=p, cin=7, cout=6, tensor_cores=tc, **cfg)
        out.append(net.forward(a).cpu().numpy())
        net.loss(target)
        net.backward()
        torch.cuda.synchronize()
        assert not net.tc_error()
        grad.append(net.grads_numpy())
    assert np.abs(out[0] - out[1]).max() <= 1.01e-2 * np.abs(out[1]).max()
    for k, g in grad[1].items():
        assert np.abs(grad[0][k] - g).max() <= 5.1e-2 * np.abs(g).max() + 1e-9, k
