"""Training-mode BatchNorm + residual + ReLU in the native kernels against the layers they stand for."""
import pytest
import torch
import torch.nn as nn

from warpconvnet_b200 import BatchNorm, Sequential, Voxels
from warpconvnet_b200.nn.functional.batch_norm import batch_norm_act, can_fuse

from conftest import rel_l2

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = {torch.float32: 4e-6, torch.float16: 2e-3, torch.bfloat16: 1.5e-2}


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n,c", [(2, 8), (3, 1024), (1000, 24), (4097, 64), (50001, 96), (30000, 256)])
@pytest.mark.parametrize("relu,with_res", [(False, False), (True, False), (True, True), (False, True)])
def test_matches_separate_layers(dtype, n, c, relu, with_res):
    g = torch.Generator().manual_seed(n + c)
    # means far from zero against the spread: the variance must not cancel
    x0 = (torch.randn(n, c, generator=g) * 0.5 + torch.randn(c, generator=g) * 3).to(dtype).to(DEV)
    r0 = torch.randn(n, c, generator=g).to(dtype).to(DEV) if with_res else None
    dy = torch.randn(n, c, generator=g).to(dtype).to(DEV)

    def build():
        torch.manual_seed(1)
        bn = nn.BatchNorm1d(c).to(DEV)
        with torch.no_grad():
            bn.weight.copy_(torch.rand(c, generator=torch.Generator().manual_seed(2)) + 0.5)
            bn.bias.copy_(torch.randn(c, generator=torch.Generator().manual_seed(3)))
        return bn, x0.clone().requires_grad_(True), r0.clone().requires_grad_(True) if with_res else None

    bn, x, r = build()
    assert can_fuse(bn, x)
    y = batch_norm_act(x, bn, relu, r)
    y.backward(dy)
    ref, xr, rr = build()
    if dtype == torch.float32:  # against fp64
        ref, xr, rr = ref.double(), xr.detach().double().requires_grad_(True), rr.detach().double().requires_grad_(True) if with_res else None
    z = ref(xr)
    z = z + rr if with_res else z
    z = torch.relu(z) if relu else z
    z.backward(dy.to(z.dtype))
    tol = TOL[dtype] * (20 if n < 10 else 1)  # a handful of rows: 1 / std amplifies every rounding
    if relu and dtype == torch.float32:
        tol = 2e-3  # values within a rounding of zero fall on the other side of the ReLU

    def close(a, b):
        return rel_l2(a.detach().double().cpu().numpy(), b.detach().double().cpu().numpy()) < tol
    assert close(y, z) and close(bn.weight.grad, ref.weight.grad) and close(bn.bias.grad, ref.bias.grad)
    assert n < 10 or close(x.grad, xr.grad)
    assert not with_res or close(r.grad, rr.grad)
    assert close(bn.running_mean, ref.running_mean) and close(bn.running_var, ref.running_var)
    assert int(bn.num_batches_tracked) == 1 and bn.running_mean._version > 0
    again = batch_norm_act(x0, build()[0], relu, r0)
    assert torch.equal(again, y)  # the same bits on every run


def test_sequential_trains_through_the_fused_layers_and_second_derivatives_work():
    n, c = 500, 16
    vox = Voxels(torch.arange(3 * n, dtype=torch.int32, device=DEV).view(n, 3), torch.randn(n, c, device=DEV), offsets=torch.tensor([0, n]))
    seq = Sequential(BatchNorm(c), nn.ReLU()).to(DEV).train()
    x = torch.randn(n, c, device=DEV, requires_grad=True)
    y = seq(vox.replace(batched_features=x)).feature_tensor
    assert "BatchNormAct" in type(y.grad_fn).__name__
    (gx,) = torch.autograd.grad((y ** 2).sum(), [x], create_graph=True)
    (ggx,) = torch.autograd.grad(gx.sum() + (gx ** 2).sum(), [x])
    xr = x.detach().clone().requires_grad_(True)
    yr = torch.relu(nn.functional.batch_norm(xr, None, None, seq[0].norm.weight, seq[0].norm.bias, True))
    (gr,) = torch.autograd.grad((yr ** 2).sum(), [xr], create_graph=True)
    (ggr,) = torch.autograd.grad(gr.sum() + (gr ** 2).sum(), [xr])
    assert rel_l2(gx.detach().cpu().numpy(), gr.detach().cpu().numpy()) < 1e-4
    assert rel_l2(ggx.cpu().numpy(), ggr.cpu().numpy()) < 1e-3


@pytest.mark.parametrize("stride,residual,relu", [(1, False, True), (1, True, True), (2, False, False)])
def test_convolution_and_norm_as_one_function(stride, residual, relu):
    """A convolution with the BatchNorm, residual and ReLU behind it in training: outputs, running statistics and every
    gradient as from the layers one by one, and a gradient of the gradient where the layers have one."""
    from warpconvnet_b200 import Sequential, SparseConv3d, Voxels
    g = torch.Generator().manual_seed(stride)
    xyz = torch.unique(torch.randint(0, 24, (4000, 3), generator=g, dtype=torch.int32), dim=0)
    n = len(xyz)
    feats = torch.randn(n, 32, generator=g).to(DEV)
    results = []
    for together in (True, False):
        torch.manual_seed(3)
        seq = Sequential(SparseConv3d(32, 64, 3 if stride == 1 else 2, stride, bias=False), nn.BatchNorm1d(64),
                         nn.ReLU() if relu and not residual else nn.Identity()).to(DEV).train()
        x = feats.clone().requires_grad_(True)
        v = Voxels(xyz.to(DEV), x, offsets=torch.tensor([0, n])).sort()
        res = torch.linspace(-1, 1, n * 64, device=DEV).view(n, 64).requires_grad_(True) if residual else None
        if together:
            y = seq(v, residual=res, final_relu=relu and residual).feature_tensor
        else:
            handle = seq[0].register_forward_hook(lambda m, a, out: None)  # a hooked layer runs by itself
            y = seq(v, residual=res, final_relu=relu and residual).feature_tensor
            handle.remove()
        w = torch.linspace(0.5, 1.5, y.numel(), device=DEV).view_as(y)
        wanted = [x, seq[0].weight, seq[1].weight, seq[1].bias] + ([res] if residual else [])
        grads = torch.autograd.grad((y * w).sum(), wanted)
        results.append([y.detach(), seq[1].running_mean.clone(), seq[1].running_var.clone(), *grads])
    for a, b in zip(*results):
        assert a.dtype == b.dtype and float((a - b).norm()) <= 1e-5 * max(1.0, float(b.norm()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_gradients_and_saved_tensors_at_any_address(dtype):
    """A gradient that is a view at an odd element of a flat buffer, and saved tensors that a hook returns as such views."""
    n, c = 300, 16
    g = torch.Generator().manual_seed(0)
    x0, r0, dy = (torch.randn(n, c, generator=g).to(dtype).to(DEV) for _ in range(3))

    def odd(t):
        return torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)

    def grads(gradient, hooks):
        bn = nn.BatchNorm1d(c).to(DEV)
        x, r = x0.clone().requires_grad_(True), r0.clone().requires_grad_(True)
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, odd if hooks else lambda t: t):
            y = batch_norm_act(x, bn, True, r)
            return torch.autograd.grad(y, [x, r, bn.weight, bn.bias], gradient)
    want = grads(dy, False)
    assert odd(dy).data_ptr() % 16
    for gradient, hooks in ((odd(dy), False), (dy, True), (odd(dy), True)):
        assert all(torch.equal(a, b) for a, b in zip(grads(gradient, hooks), want))


def test_modules_that_do_something_of_their_own_are_called_in_training():
    """Hooks on the activation, on a geometry BatchNorm or on all modules, and classes with a forward of their own."""
    from torch.nn.modules.module import register_module_forward_hook
    from warpconvnet_b200 import ReLU, SparseConv3d
    from warpconvnet_b200.examples.mink_unet import ConvTrBlock

    class Halved(SparseConv3d):
        def forward(self, *a, **kw):
            y = super().forward(*a, **kw)
            return y.replace(batched_features=y.feature_tensor * 0.5)

    class Leaky(nn.ReLU):
        def forward(self, x):
            return torch.nn.functional.leaky_relu(x, 0.1)

    g = torch.Generator().manual_seed(0)
    xyz = torch.unique(torch.randint(0, 16, (2000, 3), generator=g, dtype=torch.int32), dim=0)
    n = len(xyz)
    vox = Voxels(xyz.to(DEV), torch.randn(n, 16, generator=g).to(DEV), offsets=torch.tensor([0, n])).sort()
    for norm, act in ((nn.BatchNorm1d(16), nn.ReLU()), (BatchNorm(16), ReLU()), (BatchNorm(16), nn.Identity())):
        seq = Sequential(SparseConv3d(16, 16, 3, bias=False), norm, act).to(DEV).train()
        want = seq(vox).feature_tensor.detach()
        modules = [seq[0], norm, act, *norm.children(), *act.children()]
        for m in modules:
            seen = []
            handle = m.register_forward_hook(lambda *a: seen.append(1))
            got = seq(vox).feature_tensor
            handle.remove()
            assert seen == [1], type(m)
            assert rel_l2(got.detach().cpu().numpy(), want.cpu().numpy()) < 1e-5
        seen = []
        handle = register_module_forward_hook(lambda m, *a: seen.append(m))
        try:
            seq(vox)
        finally:
            handle.remove()
        assert all(m in seen for m in modules)
    up = ConvTrBlock(16, 16, kernel_size=2, stride=2).to(DEV).train()
    coarse = SparseConv3d(16, 16, 2, stride=2).to(DEV)(vox)
    for m in (up.conv_tr, up.norm_act, up.norm_act[0], up.norm_act[1]):
        seen = []
        handle = m.register_forward_hook(lambda *a: seen.append(1))
        up(coarse, vox)
        handle.remove()
        assert seen == [1], type(m)
    torch.manual_seed(0)
    a = Sequential(Halved(16, 16, 3, bias=False), nn.BatchNorm1d(16, eps=1.0), Leaky()).to(DEV).train()
    y = a(vox).feature_tensor
    z = nn.functional.batch_norm(a[0](vox).feature_tensor, None, None, None, None, True, 0.0, 1.0)
    assert rel_l2(y.detach().cpu().numpy(), nn.functional.leaky_relu(z, 0.1).detach().cpu().numpy()) < 1e-5


@pytest.mark.parametrize("shape", [(1, 16), (16,), ("n", 1)])
def test_residuals_that_are_broadcast_train(shape):
    from warpconvnet_b200 import SparseConv3d
    g = torch.Generator().manual_seed(0)
    xyz = torch.unique(torch.randint(0, 16, (2000, 3), generator=g, dtype=torch.int32), dim=0)
    n = len(xyz)
    vox = Voxels(xyz.to(DEV), torch.randn(n, 16, generator=g).to(DEV), offsets=torch.tensor([0, n]))
    res = torch.randn([n if s == "n" else s for s in shape], generator=g).to(DEV).requires_grad_(True)
    for seq in (Sequential(SparseConv3d(16, 16, 3, bias=False), nn.BatchNorm1d(16)), Sequential(nn.BatchNorm1d(16))):
        seq = seq.to(DEV).train()
        y = seq(vox, residual=res, final_relu=True).feature_tensor
        want = torch.relu(seq(vox).feature_tensor + res)
        assert rel_l2(y.detach().cpu().numpy(), want.detach().cpu().numpy()) < 1e-6
        (a,), (b,) = torch.autograd.grad(y.sum(), [res]), torch.autograd.grad(want.sum(), [res])
        assert a.shape == res.shape and rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 1e-5


def test_captured_steps_do_not_depend_on_one_another():
    """Of two graphs over the same memory pool the one captured last is replayed first (and the other never): nothing it
    reads may be left to the first one to initialise."""
    n, c = 5000, 32
    x = torch.randn(n, c, device=DEV)
    bn = nn.BatchNorm1d(c).to(DEV)
    want = batch_norm_act(x, bn, True)
    pool = torch.cuda.graph_pool_handle()

    def captured(fn):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, pool=pool):
            out = fn()
        return graph, out
    junk, blocks = captured(lambda: [torch.full((131072,), 12345, dtype=torch.int32, device=DEV) for _ in range(16)])
    junk.replay()
    torch.cuda.synchronize()
    del blocks
    first = captured(lambda: batch_norm_act(x, bn, True))
    second = captured(lambda: batch_norm_act(x, bn, True))
    for _ in range(2):
        second[0].replay()
        assert torch.equal(second[1], want)
    del first, second, junk


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("n,c", [(2, 8), (7, 24), (50001, 64), (18945, 96), (200000, 16), (30000, 1024)])
@pytest.mark.parametrize("at", [0, -1])
def test_variance_keeps_its_precision_beside_a_large_value(dtype, n, c, at):
    """One row far from all others, the first or the last one: the variance within a few dozen fp32 roundings,
    the mean within as many of the spread."""
    x = torch.randn(n, c, generator=torch.Generator().manual_seed(c)).to(dtype)
    x[at] = 1000.0
    bn = nn.BatchNorm1d(c, momentum=1.0).to(DEV)
    with torch.no_grad():
        batch_norm_act(x.to(DEV), bn)
    xd = x.double()
    mean, var = xd.mean(0), xd.var(0)
    assert float((bn.running_mean.cpu().double() - mean).abs().max()) < 1e-6 * float(var.sqrt().min())
    assert rel_l2(bn.running_var.cpu().numpy(), var.numpy()) < 2e-6


def test_infinite_and_missing_values_reach_the_statistics():
    """A channel with an infinity or a NaN has no variance; the others are untouched (as with nn.BatchNorm1d)."""
    n, c = 1000, 16
    x = torch.randn(n, c, device=DEV)
    clean = batch_norm_act(x, nn.BatchNorm1d(c).to(DEV)).detach()
    x[n // 2, 3], x[0, 5], x[n - 1, 7] = float("inf"), float("-inf"), float("nan")
    y = batch_norm_act(x, nn.BatchNorm1d(c).to(DEV)).detach()
    bad = torch.zeros(c, dtype=torch.bool, device=DEV)
    bad[[3, 5, 7]] = True
    assert torch.isnan(y[:, bad]).all() and torch.equal(y[:, ~bad], clean[:, ~bad])


@pytest.mark.parametrize("which", ["running_mean", "running_var", "weight", "bias", "num_batches_tracked"])
def test_parameters_that_the_kernel_does_not_read_take_the_module(which):
    """Every second element of a wider buffer, or a counter of another type: computed by nn.BatchNorm1d as before."""
    n, c = 200, 16
    x = torch.randn(n, c, device=DEV)

    def build(strided):
        g = torch.Generator().manual_seed(0)
        bn = nn.BatchNorm1d(c).to(DEV)
        for name in ("running_mean", "running_var", "weight", "bias"):
            v = torch.rand(c, generator=g).to(DEV) + 0.5
            if strided and name == which:
                wide = torch.zeros(2 * c, device=DEV)
                wide[::2] = v
                v = wide[::2]
            getattr(bn, name).data = v
        if strided and which == "num_batches_tracked":
            bn.num_batches_tracked = bn.num_batches_tracked.cpu()
        return Sequential(bn).train()
    vox = Voxels(torch.arange(3 * n, dtype=torch.int32, device=DEV).view(n, 3), x, offsets=torch.tensor([0, n]))
    a, b = build(True), build(False)
    assert not can_fuse(a[0], x) and can_fuse(b[0], x)
    ya, yb = a(vox).feature_tensor, b(vox).feature_tensor
    assert rel_l2(ya.detach().cpu().numpy(), yb.detach().cpu().numpy()) < 1e-6
    for p, q in zip(a[0].buffers(), b[0].buffers()):
        assert rel_l2(p.cpu().numpy(), q.cpu().numpy()) < 1e-6
