"""GPU parity of pooling over kernel maps: ``sparse_reduce`` / ``sparse_unpool`` and the
``reduce_and_stride`` mode of the convolution against the oracle's restatement of the reference."""
import numpy as np
import pytest
import torch

from oracle import kernel_map as km
from oracle import sparse_conv as osc
from warpconvnet_b200 import (SPARSE_CONV_FWD_ALGO_MODE as ALGO, STRIDED_CONV_MODE, SparseMaxPool, SparseUnpool, Voxels,
                              sparse_reduce, sparse_unpool, spatially_sparse_conv)
from warpconvnet_b200._native import check_device_status
from warpconvnet_b200.datasets import synthetic

from conftest import rel_l2

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _scene(n, c, seed, dtype=torch.float32):
    scenes = [synthetic.room_scene(n, 0.04, seed + i, "sample") - 17 for i in range(2)]
    coords, offsets = synthetic.batch_scenes(scenes)
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(len(coords), c, generator=g).to(dtype)
    vox = Voxels(torch.from_numpy(coords[:, 1:].copy()).to(DEV), x.to(DEV), offsets=torch.from_numpy(offsets))
    return coords.astype(np.int32), x, vox


@pytest.mark.parametrize("reduction", ["max", "min", "mean", "sum", "mul", "var", "std"])
@pytest.mark.parametrize("c", [7, 32])
def test_sparse_reduce_matches_oracle(reduction, c):
    coords, x, vox = _scene(6000, c, 61)
    if reduction == "mul":
        x = x * 0.5 + 1.0
        vox = vox.replace(batched_features=x.to(DEV))
    out = sparse_reduce(vox, kernel_size=2, stride=2, reduction=reduction)
    check_device_status(DEV)
    ref_c, ref_off = km.stride_coords(coords, (2, 2, 2))
    i, o, f, _ = km.generate_kernel_map(coords, ref_c, (2, 2, 2), (2, 2, 2))
    want = osc.window_reduce(x.numpy(), i, o, len(ref_c), reduction)
    assert np.array_equal(out.batch_indexed_coordinates.cpu().numpy(), ref_c)
    assert np.array_equal(out.offsets.numpy(), ref_off)
    assert out.tensor_stride == (2, 2, 2)
    tol = 1e-4 if reduction in ("var", "std") else 1e-6
    assert rel_l2(out.feature_tensor.cpu().numpy(), want) < tol
    if reduction in ("max", "min"):
        assert np.array_equal(out.feature_tensor.cpu().numpy(), want.astype(np.float32))


def test_overlapping_windows_fp16_and_random():
    coords, x, vox = _scene(5000, 16, 62, torch.float16)
    out = sparse_reduce(vox, kernel_size=3, stride=2, reduction="max")
    ref_c, _ = km.stride_coords(coords, (2, 2, 2))
    i, o, f, _ = km.generate_kernel_map(coords, ref_c, (2, 2, 2), (3, 3, 3))
    want = osc.window_reduce(x.float().numpy(), i, o, len(ref_c), "max")
    assert np.array_equal(out.feature_tensor.float().cpu().numpy(), want.astype(np.float32))
    # random: every output row is one of the rows of its window
    rnd = sparse_reduce(vox, kernel_size=2, stride=2, reduction="random").feature_tensor.float().cpu().numpy()
    i2, o2, _, _ = km.generate_kernel_map(coords, ref_c, (2, 2, 2), (2, 2, 2))
    lo = osc.window_reduce(x.float().numpy(), i2, o2, len(ref_c), "min")
    hi = osc.window_reduce(x.float().numpy(), i2, o2, len(ref_c), "max")
    assert np.all(rnd >= lo - 1e-6) and np.all(rnd <= hi + 1e-6)
    check_device_status(DEV)


@pytest.mark.parametrize("concat", [True, False])
def test_unpool_copies_parents_back(concat):
    coords, x, vox = _scene(4000, 5, 63)
    pooled = SparseMaxPool(2, 2)(vox)
    up = SparseUnpool(2, 2, concat_unpooled_st=concat)(pooled, vox)
    ref_c, _ = km.stride_coords(coords, (2, 2, 2))
    i, o, f, _ = km.generate_kernel_map(coords, ref_c, (2, 2, 2), (2, 2, 2))
    parent = np.empty(len(coords), dtype=np.int64)
    parent[i] = o
    want = pooled.feature_tensor.cpu().numpy()[parent]
    got = up.feature_tensor.cpu().numpy()
    if concat:
        assert got.shape[1] == 10 and np.array_equal(got[:, :5], x.numpy()) and np.array_equal(got[:, 5:], want)
    else:
        assert np.array_equal(got, want)
    assert up.coordinate_tensor.shape[0] == len(coords)


def test_reduce_and_stride_convolution():
    """stride_mode=reduce_and_stride: pool the stride window (max), then a stride-1 convolution on the
    pooled tensor (warpconvnet/nn/functional/sparse_conv.py:1753-1767)."""
    coords, x, vox = _scene(5000, 8, 64)
    g = torch.Generator().manual_seed(3)
    w = torch.randn(27, 8, 12, generator=g) * 0.2
    with torch.no_grad():
        y = spatially_sparse_conv(vox, w.to(DEV), 3, stride=2, stride_mode=STRIDED_CONV_MODE.REDUCE_AND_STRIDE,
                                  stride_reduce="max", fwd_algo=ALGO.IMPLICIT_GEMM)
    ref_c, _ = km.stride_coords(coords, (2, 2, 2))
    i, o, f, _ = km.generate_kernel_map(coords, ref_c, (2, 2, 2), (2, 2, 2))
    pooled = osc.window_reduce(x.numpy(), i, o, len(ref_c), "max").astype(np.float32)
    i3, o3, f3, iden = km.generate_kernel_map(ref_c, ref_c, (1, 1, 1), (3, 3, 3))
    want = osc.explicit_gemm_forward(torch.from_numpy(pooled), w, i3, o3, f3, iden, len(ref_c)).numpy()
    assert np.array_equal(y.batch_indexed_coordinates.cpu().numpy(), ref_c)
    assert y.tensor_stride == (2, 2, 2)
    assert rel_l2(y.feature_tensor.cpu().numpy(), want) < 1e-4
    check_device_status(DEV)


@pytest.mark.parametrize("reduction", ["max", "min", "mean", "sum"])
@pytest.mark.parametrize("dtype,c,ksize", [(torch.float32, 4, 2), (torch.float32, 7, 3), (torch.float16, 8, 2),
                                           (torch.bfloat16, 24, 3), (torch.float16, 9, 2), (torch.float16, 8, 7)])
def test_pooling_gradients_of_every_width(reduction, dtype, c, ksize):
    """The gradient kernel at whole and odd channel counts, at windows of 8, 27 and 343 offsets (one and two bytes per
    arg-extremum), overlapping or not, with ties, against the reduction's definition over the kernel map."""
    coords, x, vox = _scene(1500, c, 63, dtype)
    x = (x * 2).round() / 2  # many equal values: the first offset takes the gradient
    xg = x.to(DEV).requires_grad_(True)
    out = sparse_reduce(vox.replace(batched_features=xg), kernel_size=ksize, stride=2, reduction=reduction).feature_tensor
    g = torch.randn(out.shape, generator=torch.Generator().manual_seed(64)).to(dtype)
    (got,) = torch.autograd.grad(out, [xg], g.to(DEV))
    ref_c, _ = km.stride_coords(coords, (2, 2, 2))
    i, o, f, _ = km.generate_kernel_map(coords, ref_c, (2, 2, 2), (ksize,) * 3)
    k = np.repeat(np.arange(len(f) - 1), np.diff(f))
    want = np.zeros((len(coords), c))
    count = np.bincount(o, minlength=len(ref_c))
    xs, gs = x.double().numpy(), g.double().numpy()
    if reduction in ("max", "min"):
        s = 1.0 if reduction == "max" else -1.0
        top = np.full((len(ref_c), c), -np.inf)
        at = np.full((len(ref_c), c), -1)
        for p in np.argsort(k, kind="stable"):
            beyond = s * xs[i[p]] > top[o[p]]
            top[o[p]][beyond] = s * xs[i[p]][beyond]
            at[o[p]][beyond] = i[p]
        for ch in range(c):
            np.add.at(want[:, ch], at[:, ch], gs[:, ch])
    else:
        np.add.at(want, i, gs[o] / (count[o][:, None] if reduction == "mean" else 1.0))
    check_device_status(DEV)
    assert rel_l2(got.double().cpu().numpy(), want) < {torch.float32: 1e-6, torch.float16: 1e-3, torch.bfloat16: 8e-3}[dtype]


@pytest.mark.parametrize("reduction", ["max", "min", "mean", "sum"])
@pytest.mark.parametrize("ksize", [2, 3])
def test_pooling_has_second_derivatives(reduction, ksize):
    """The gradient of a gradient, through the definition over the kernel map in fp64."""
    coords, x, vox = _scene(800, 5, 67)
    x = vox.feature_tensor.clone().requires_grad_(True)
    out = sparse_reduce(vox.replace(batched_features=x), kernel_size=ksize, stride=2, reduction=reduction)
    from warpconvnet_b200 import generate_kernel_map
    nbr = generate_kernel_map(vox.batch_indexed_coordinates.contiguous(), out.batch_indexed_coordinates.contiguous(), (2, 2, 2),
                              (ksize,) * 3).neighbor_table(len(out)).long()
    xd = x.detach().double().requires_grad_(True)
    have = (nbr >= 0).unsqueeze(2)
    rows = xd[nbr.clamp(min=0)]
    if reduction in ("max", "min"):
        s = 1.0 if reduction == "max" else -1.0
        window = torch.where(have, s * rows, -torch.inf)
        want = s * window.gather(0, window.argmax(0, keepdim=True))[0]
    else:
        want = torch.where(have, rows, 0.0).sum(0)
        want = want / have.sum(0) if reduction == "mean" else want

    def second(y, x0):
        (gx,) = torch.autograd.grad((y ** 3).sum(), [x0], create_graph=True)
        (ggx,) = torch.autograd.grad((gx ** 2).sum(), [x0])
        return gx.detach(), ggx
    for a, b in zip(second(out.feature_tensor, x), second(want, xd)):
        assert rel_l2(a.double().cpu().numpy(), b.cpu().numpy()) < 1e-5
    check_device_status(DEV)


@pytest.mark.parametrize("reduction", ["max", "min"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_extremum_gradients_over_repeated_voxels(reduction, dtype):
    """Pooling at stride 1 over repeated voxels: the outputs of a voxel's copies all take the same input row, whose
    gradient is the sum of theirs."""
    coords, x, _ = _scene(1500, 8, 65, dtype)
    coords = np.concatenate([coords[coords[:, 0] == 0], coords[coords[:, 0] == 0][::3]])
    n = len(coords)
    g = torch.Generator().manual_seed(66)
    x = torch.randn(n, 8, generator=g).to(dtype).to(DEV).requires_grad_(True)
    vox = Voxels(torch.from_numpy(coords[:, 1:].copy()).to(DEV), x, offsets=torch.tensor([0, n]))
    out = sparse_reduce(vox, kernel_size=3, stride=1, reduction=reduction).feature_tensor
    dy = torch.randn(out.shape, generator=g).to(dtype).to(DEV)
    (got,) = torch.autograd.grad(out, [x], dy)
    from warpconvnet_b200 import generate_kernel_map
    rows = vox.batch_indexed_coordinates.contiguous()
    nbr = generate_kernel_map(rows, rows, (1, 1, 1), (3, 3, 3)).neighbor_table(n).long()
    xd = x.detach().double().requires_grad_(True)
    s = 1.0 if reduction == "max" else -1.0
    window = torch.where((nbr >= 0).unsqueeze(2), s * xd[nbr.clamp(min=0)], -torch.inf)
    want = s * window.gather(0, window.argmax(0, keepdim=True))[0]   # (the first of equal values)
    (ref,) = torch.autograd.grad(want, [xd], dy.double())
    assert torch.equal(out.detach().double(), want.detach())
    assert rel_l2(got.double().cpu().numpy(), ref.cpu().numpy()) < (1e-6 if dtype == torch.float32 else 1e-3)
    check_device_status(DEV)
