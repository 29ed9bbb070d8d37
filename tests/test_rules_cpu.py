"""Which fp32 problems go to the tensor cores: the byte queries that the callers ask (no GPU needed)."""
import pytest
import torch

from warpconvnet_b200._native import query_bytes


@pytest.mark.parametrize("problem,taken", [
    ((100000, 100000, 27, 64, 64), True),
    ((1000000, 250000, 8, 64, 64), True), ((1000000, 250000, 8, 32, 32), True),          # strided layers keep them
    # a small part of the output rows: planes of all input rows take longer than the launch
    ((1000000, 62500, 27, 64, 64), True), ((1000000, 15625, 27, 64, 64), False), ((1000000, 15625, 27, 128, 128), False),
    ((1000000, 2000, 27, 64, 64), False), ((100000, 6250, 27, 64, 64), True), ((1000000, 1 << 40, 27, 64, 64), True),
    # rows of 16 channels become planes of 32
    ((100000, 100000, 8, 16, 16), True), ((1000000, 1000000, 8, 16, 16), False), ((300000, 300000, 27, 16, 16), False),
    ((300000, 300000, 27, 32, 16), True), ((1000000, 1000000, 8, 32, 32), True),
])
def test_layers(problem, taken):
    assert (query_bytes("wcn_conv_f32_workspace_bytes", *problem) > 0) == taken


@pytest.mark.parametrize("problem,taken", [((100000, 100000, 27, 64, 64), True), ((1000000, 200000, 27, 64, 64), True),
                                           ((1000000, 15625, 27, 64, 64), False), ((100000, 6250, 27, 64, 64), True)])
def test_weight_gradients(problem, taken):
    assert (query_bytes("wcn_conv_wgrad_f32_workspace_bytes", *problem) > 0) == taken


def test_what_a_backward_pass_asks_for():
    """``_asked_for`` of a function's inputs: leaves and others, under ``backward`` and under ``grad`` of some of them."""
    from warpconvnet_b200.nn.functional.sparse_conv import _asked_for
    said = []

    class Sum(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x, w, b):
            return x + w + b

        @staticmethod
        def backward(ctx, g):
            said.append((_asked_for(ctx.next_functions[:2]), _asked_for(ctx.next_functions[2:])))
            return g, g, g

    x, w, b = (torch.ones(2, requires_grad=True) for _ in range(3))
    y = Sum.apply(x, w, b).sum()
    for inputs in ([b], [w], [x, b]):
        torch.autograd.grad(y, inputs, retain_graph=True)
    y.backward(retain_graph=True)
    y.backward(inputs=[b])
    assert said == [(False, True), (True, False), (True, True), (True, True), (False, True)]
    said.clear()
    inner = x * 2
    y = Sum.apply(inner, w.detach(), b).sum()
    for inputs in ([b], [inner], [x]):
        torch.autograd.grad(y, inputs, retain_graph=True)
    y.backward()
    assert said == [(False, True), (True, False), (True, False), (True, True)]
