"""Pieces of the learned guess's pass on their own: paired products against
the two products one after the other, channel sums against FP64 sums, and the
bias / activation passes in their float4 and scalar forms against PyTorch.

Tolerances.  Pairs: none (both forms round the same operands to the same
tensor-core products, and alpha and beta are powers of two, so that however
the epilogue is contracted it rounds alike).  Channel sums: the sum is FP64,
so only the rounding of the result, and of beta * out + sum, to FP32 is left:
3 units of 2^-24 of the magnitudes added.  Bias: one FP32 addition, exact.
Activation and its derivative: FP32 evaluations against FP64, 2^-19 (the
arguments reach 4, a handful of FP32 operations each)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# batch, M, N, K, A strides, B strides, C strides, alpha, beta, kind
#   sum: C += A0 B0 + A1 B1; split: C0 = A B0, C1 = A B1; left: the shared
#   operand is the left one (the transposed form), C0 = A0 B, C1 = A1 B
PAIRS = {
    "sum-two-row-tiles": (5, 64, 16, 64, (4096, 64, 1), (0, 16, 1), (1024, 16, 1), 1.0, 0.0, "sum"),
    "sum-short-k-onto-c": (6, 64, 64, 16, (2048, 16, 1), (0, 64, 1), (4096, 64, 1), 1 / 4096, 1.0, "sum"),
    "sum-ragged": (3, 37, 21, 70, (37 * 71, 71, 1), (0, 21, 1), (37 * 21, 21, 1), 0.5, 1.0, "sum"),
    "sum-left": (7, 24, 12, 9, (0, 9, 1), (1, 12 * 7, 7), (24 * 12, 12, 1), 1.0, 0.0, "sum"),
    "split-two-column-tiles": (2, 40, 100, 130, (40 * 132, 132, 1), (0, 100, 1), (4000, 100, 1), 2.0, 0.0, "split"),
    "split-k-contiguous": (4, 50, 16, 64, (3200, 64, 1), (0, 1, 64), (800, 16, 1), 1.0, 1.0, "split"),
    "split-k-contiguous-ragged": (2, 33, 36, 70, (33 * 72, 72, 1), (0, 1, 72), (33 * 36, 36, 1), 1.0, 0.0, "split"),
    "left-interleaved": (9, 16, 20, 128, (0, 128, 1), (128 * 20, 20, 1), (1, 20 * 18, 18), 1.0, 0.0, "left"),
    "left-transposed": (3, 18, 8, 100, (0, 1, 18), (800, 8, 1), (144, 8, 1), 1.0, 0.0, "left"),
    "one-element": (1, 1, 1, 1, (1, 1, 1), (0, 1, 1), (1, 1, 1), 2.0, 0.0, "sum"),
}


def _span(batch, rows, cols, s):
    return 1 + (batch - 1) * s[0] + (rows - 1) * s[1] + (cols - 1) * s[2]


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("name", list(PAIRS))
def test_paired_products_are_the_two_products(name):
    from fortress_b200 import fno as FN
    L = FN.lib()
    batch, M, N, K, sA, sB, sC, alpha, beta, kind = PAIRS[name]
    gen = torch.Generator("cuda").manual_seed(M * 131 + K)

    def rand(n):
        return torch.randn(n, device="cuda", generator=gen)

    A = [rand(_span(batch, M, K, sA)) for _ in range(2)]
    B = [rand(_span(batch, K, N, sB)) for _ in range(2)]
    C = [rand(_span(batch, M, N, sC)) for _ in range(2)]
    if kind == "split":
        A[1] = A[0]
    elif kind == "left":
        B[1] = B[0]
    else:
        C[1] = C[0]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    want = [C[0].clone()]
    want.append(want[0] if kind == "sum" else C[1].clone())
    for q in range(2):
        assert 0 == L.fno_gemm_tc(batch, M, N, K, alpha, _p(A[q]), 0, *sA, _p(B[q]), *sB,
                                  1.0 if kind == "sum" and q else beta, _p(want[q]), *sC, _p(err), st)
    assert 0 == L.fno_gemm_tc2(batch, M, N, K, alpha, _p(A[0]), _p(A[1]), *sA, _p(B[0]), _p(B[1]), *sB, beta,
                               _p(C[0]), _p(C[1]), *sC, _p(err), st)
    torch.cuda.synchronize()
    assert err.item() == 0
    assert torch.equal(C[0], want[0]) and torch.equal(C[1], want[1])


def test_a_pair_that_shares_nothing_is_refused():
    from fortress_b200 import fno as FN
    t = [torch.zeros(64, device="cuda") for _ in range(6)]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = FN.lib().fno_gemm_tc2(1, 8, 8, 8, 1.0, _p(t[0]), _p(t[1]), 64, 8, 1, _p(t[2]), _p(t[3]), 64, 8, 1, 0.0,
                               _p(t[4]), _p(t[5]), 64, 8, 1, _p(err), None)
    assert rc != 0


# batch, planes per channel, n (M = N), K, beta, act, offset of H in elements
@pytest.mark.parametrize("batch,per,n,K,beta,act,off", [(12, 4, 64, 16, 1.0, 1, 0), (6, 2, 37, 9, 1.0, 1, 0), (4, 4, 20, 16, 0.0, 0, 0),
                                                        (6, 3, 32, 16, 1.0, 1, 1), (1, 1, 1, 1, 1.0, 1, 0)])
def test_pair_with_bias_and_activation_is_the_two_passes(batch, per, n, K, beta, act, off):
    from fortress_b200 import fno as FN
    L = FN.lib()
    gen = torch.Generator("cuda").manual_seed(n * 7 + K)
    A = [torch.randn(batch * n * K, device="cuda", generator=gen) for _ in range(2)]
    B = [torch.randn(K * n, device="cuda", generator=gen) for _ in range(2)]
    C = torch.randn(batch * n * n, device="cuda", generator=gen)
    bias = torch.randn(batch // per, device="cuda", generator=gen)
    H, err = torch.zeros(C.numel() + off, device="cuda")[off:], torch.zeros(1, dtype=torch.int32, device="cuda")
    want, wanth = C.clone(), torch.zeros_like(C)
    sA, sB, sC, S = (n * K, K, 1), (0, n, 1), (n * n, n, 1), per * n * n
    assert 0 == L.fno_gemm_tc2(batch, n, n, K, 0.25, _p(A[0]), _p(A[1]), *sA, _p(B[0]), _p(B[1]), *sB, beta, _p(want),
                               _p(want), *sC, _p(err), None)
    assert 0 == L.fno_bias_act(_p(want), _p(wanth), _p(bias), batch // per, S, want.numel(), act, None)
    assert 0 == L.fno_gemm_tc2_act(batch, n, n, K, 0.25, _p(A[0]), _p(A[1]), *sA, _p(B[0]), _p(B[1]), *sB, beta, _p(C), *sC,
                                   _p(bias), batch // per, S, act, _p(H), _p(err), None)
    torch.cuda.synchronize()
    assert err.item() == 0
    # the same operations in the same order; the activation is compiled twice
    # (products may fuse differently): a few units of 2^-24 of values up to 64
    assert torch.equal(C, want)
    assert (H - wanth).abs().max().item() <= (0.0 if act == 0 else 2.0 ** -24 * 64 * 8)


@pytest.mark.parametrize("B,C,S,off", [
    (1, 1, 1, 0), (7, 33, 1, 0), (300, 1000, 1, 0),          # S = 1: channels past a block, batch not a multiple of 8
    (1, 3, 2, 0), (2, 32, 37, 0), (3, 5, 4096, 0),           # fewer points than blocks, ragged and full slices
    (2, 3, 1027, 0), (2, 2, 8196, 1),                        # rows off a 16-byte boundary
])
@pytest.mark.parametrize("beta", [0.0, 1.0])
def test_channel_sums(B, C, S, off, beta):
    from fortress_b200 import fno as FN
    gen = torch.Generator("cuda").manual_seed(C * S)
    x = torch.randn(B * C * S + off, device="cuda", generator=gen)[off:]
    out = torch.randn(C, device="cuda", generator=gen)
    xs = x.double().view(B, C, S)
    want = beta * out.double() + xs.sum((0, 2))
    bound = 3 * 2.0 ** -24 * (want.abs() + xs.sum((0, 2)).abs() + out.double().abs())
    assert 0 == FN.lib().fno_channel_sum(_p(out), _p(x), B, C, S, beta, None)
    torch.cuda.synchronize()
    assert bool(((out.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("C,S,B,off", [(3, 8, 2, 0), (5, 7, 3, 0), (2, 64, 1, 1), (1, 1, 1, 0), (32, 1024, 3, 0)])
def test_bias_and_activation_forms(C, S, B, off):
    from fortress_b200 import fno as FN
    L = FN.lib()
    n = B * C * S
    gen = torch.Generator("cuda").manual_seed(n)
    z = (torch.rand(n + off, device="cuda", generator=gen)[off:] - 0.5) * 6
    h = torch.zeros(n + off, device="cuda")[off:]
    bias = torch.rand(C, device="cuda", generator=gen)
    want = (z.view(B, C, S) + bias.view(1, C, 1)).reshape(-1)
    assert 0 == L.fno_bias_act(_p(z), _p(h), _p(bias), C, S, n, 1, None)
    torch.cuda.synchronize()
    assert torch.equal(z, want)
    zd = want.double().requires_grad_()
    g = torch.nn.functional.gelu(zd, approximate="tanh")
    assert (g.detach() - h.double()).abs().max().item() <= 4 * 2.0 ** -19
    dh, dz = torch.randn(n + off, device="cuda", generator=gen)[off:], torch.empty(n + off, device="cuda")[off:]
    g.backward(dh.double())
    assert 0 == L.fno_act_bwd(_p(dz), _p(dh), _p(z), n, None)
    torch.cuda.synchronize()
    assert ((dz.double() - zd.grad).abs() <= 4 * 2.0 ** -19 * (1 + dh.double().abs())).all()
