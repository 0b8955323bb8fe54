"""The network's fused passes at the batch sizes where their tiles change, against the
single steps (im2col and the GEMM) they replace and against PyTorch.

A forward pass multiplies and adds in the same order as the single steps, so its
activations round alike and its logits are the same bits; the gradients, which round
intermediate values to bf16, are compared with fp32 autograd at 3e-2 relative L2.
"""

from __future__ import annotations

import pytest

from test_gpu_proposal import _bf, _torch_net, torch  # noqa: F401  (torch is a fixture)

pytestmark = pytest.mark.gpu


def _stepwise(torch, net, x):
    from cuperiod_b200.proposal import (CHANNELS, HIDDEN, IN_CHANNELS, N_BINS, N_CLASSES, N_CONV,
                                        kp)
    ops, B = net.ops, x.shape[0]
    act, L, C = x.contiguous(), N_BINS, IN_CHANNELS
    for layer in range(N_CONV):
        k, R = kp(layer), B * (L // 2)
        col = torch.empty((R, k), dtype=torch.bfloat16, device="cuda")
        ops.im2col(act, col, B, L, C, k)
        y = torch.empty((R, CHANNELS), dtype=torch.bfloat16, device="cuda")
        ops.gemm(col, net.half[layer], y, M=R, N=CHANNELS, K=k, lda=k, ldb=k, ldo=CHANNELS,
                 bias=net.master[N_CONV + layer], relu=True)
        act, L, C = y, L // 2, CHANNELS
    flat = CHANNELS * L
    h = torch.empty((B, HIDDEN), dtype=torch.bfloat16, device="cuda")
    ops.gemm(act, net.half[2 * N_CONV], h, M=B, N=HIDDEN, K=flat, lda=flat, ldb=flat, ldo=HIDDEN,
             bias=net.master[2 * N_CONV + 1], relu=True)
    out = torch.empty((B, N_CLASSES), dtype=torch.float32, device="cuda")
    ops.gemm(h, net.half[2 * N_CONV + 2], out, M=B, N=N_CLASSES, K=HIDDEN, lda=HIDDEN, ldb=HIDDEN,
             ldo=N_CLASSES, mode=1, bias=net.master[2 * N_CONV + 3])
    ops.check()
    return out


@pytest.mark.parametrize("B", [1, 2, 3, 127, 129, 301])
def test_forward_equals_the_single_steps(torch, B):
    from cuperiod_b200.proposal import IN_CHANNELS, N_BINS, ProposalNet, Weights
    net = ProposalNet(Weights.init(seed=5))
    x = _bf(torch, (B, N_BINS, IN_CHANNELS), B)
    got = net.forward(x)
    net.ops.check()
    assert torch.equal(got, _stepwise(torch, net, x))


def test_forward_of_an_array_off_four_bytes(torch):
    from cuperiod_b200.proposal import IN_CHANNELS, N_BINS, ProposalNet, Weights
    net = ProposalNet(Weights.init(seed=5))
    n = 5 * N_BINS * IN_CHANNELS
    x = _bf(torch, (n + 1,), 3)[1:].view(5, N_BINS, IN_CHANNELS)
    assert x.data_ptr() % 4 == 2
    got = net.forward(x)
    net.ops.check()
    assert torch.equal(got, _stepwise(torch, net, x.clone()))


@pytest.mark.parametrize("B", [8, 24, 136])
def test_gradients_match_autograd(torch, B):
    from cuperiod_b200.proposal import IN_CHANNELS, N_BINS, N_CLASSES, ProposalNet, Weights
    w = Weights.init(seed=B)
    net = ProposalNet(w, train=True)
    x = _bf(torch, (B, N_BINS, IN_CHANNELS), 2 * B)
    labels = torch.full((B,), 700, dtype=torch.int32, device="cuda")
    d, _ = net.loss_and_grad(net.forward(x), labels, side=0.1)
    net.zero_grad()
    net.backward(d)
    once = [g.clone() for g in net.g]
    net.backward(d)                     # adds to the gradients
    net.ops.check()
    params, fwd = _torch_net(torch, w)
    target = torch.zeros((B, N_CLASSES), device="cuda")
    target[:, 699:702] = torch.tensor([0.1, 0.8, 0.1], device="cuda")
    loss = -(target * torch.log_softmax(fwd(x), dim=1)).sum() / B
    loss.backward()
    for g, g1, p in zip(net.g, once, params):
        assert float((g1 - p.grad).norm()) <= 3e-2 * float(p.grad.norm())
        torch.testing.assert_close(g, 2.0 * g1, rtol=1e-5, atol=1e-6 * float(g1.abs().max()))


def test_backward_refuses_a_batch_that_is_no_multiple_of_eight(torch):
    from cuperiod_b200._lib import EngineError
    from cuperiod_b200.proposal import IN_CHANNELS, N_BINS, N_CLASSES, ProposalNet, Weights
    net = ProposalNet(Weights.init(seed=1), train=True)
    net.forward(_bf(torch, (4, N_BINS, IN_CHANNELS), 1))
    with pytest.raises(EngineError):
        net.backward(torch.zeros((4, N_CLASSES), dtype=torch.bfloat16, device="cuda"))
