"""GPU tests of the fp32 layers' tensor-core kernels, of a training layer's bias and of the order in which the
half-precision convolution takes its units."""
import pytest
import torch

from warpconvnet_b200 import ConvEpilogue, IntSearchResult, SparseConv3d
from warpconvnet_b200._native import CONV_SIMT, CONV_TCGEN05, check_device_status
from warpconvnet_b200.nn.functional.sparse_conv import sparse_conv_fused

from conftest import rel_l2
from test_conv_gpu import make_voxels, room_rows

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _random_map(K, n, num_in, g):
    present = torch.rand(K, n, generator=g, device=DEV) < torch.rand(n, generator=g, device=DEV) ** 2
    nbr = torch.randint(0, num_in, (K, n), generator=g, device=DEV, dtype=torch.int32)
    return IntSearchResult.from_neighbor_table(torch.where(present, nbr, torch.full((), -1, dtype=torch.int32, device=DEV)), num_in)


@pytest.mark.parametrize("K,n,num_in,c_in,c_out", [(27, 1, 1, 64, 32), (27, 129, 500, 52, 48), (8, 2000, 4000, 36, 144), (8, 700, 700, 32, 32), (1, 13000, 13000, 128, 96), (27, 300, 300, 64, 64), (27, 14000, 14000, 20, 16),
                                                   (27, 9472, 9000, 32, 128), (27, 9473, 9473, 96, 112), (27, 18945, 18945, 32, 32),
                                                   (27, 70000, 70000, 64, 64), (3, 700, 600, 160, 256)])
def test_fp32_on_the_tensor_cores_is_closer_to_exact_sums(K, n, num_in, c_in, c_out):
    """Offsets divided among a cluster and not, whole and partial row tiles, column blocks, channels that do not fill a
    slice, rows apart, every part of the epilogue: against sums in 64 bits.  What is dropped of a product is below 2^-25
    of it and an accumulator adds 32 channels before it is rounded: 3e-7 is twice the largest error measured."""
    g = torch.Generator(device=DEV).manual_seed(n)
    kmap = _random_map(K, n, num_in, g)
    nbr = kmap.neighbor_table(n)
    wide = torch.randn(num_in, c_in + 4, generator=g, device=DEV)
    x = wide[:, 4:]
    w = torch.randn(K, c_in, c_out, generator=g, device=DEV) * (K * c_in) ** -0.5
    res, scale, shift = torch.randn(n, c_out, generator=g, device=DEV), torch.rand(c_out, generator=g, device=DEV) + 0.5, torch.randn(c_out, generator=g, device=DEV)
    want = torch.zeros(n, c_out, dtype=torch.float64, device=DEV)
    for k in range(K):
        m = (nbr[k] >= 0).nonzero()[:, 0]
        want[m] += x[nbr[k, m].long()].double() @ w[k].double()
    got = sparse_conv_fused(x, w, kmap, n)
    again = sparse_conv_fused(x, w, kmap, n, tile_order=True)
    simt = sparse_conv_fused(x, w, kmap, n, algo=CONV_SIMT)
    check_device_status(DEV)
    error = lambda y: float((y.double() - want).norm() / want.norm().clamp(min=1e-30))
    assert error(got) < 3e-7 and error(again) < 3e-7
    if n * c_out > 30000:
        assert error(got) <= error(simt)
    full = sparse_conv_fused(x, w, kmap, n, epilogue=ConvEpilogue(scale=scale, shift=shift, residual=res, relu=True))
    want = (want * scale.double() + shift.double() + res.double()).clamp(min=0)
    assert error(full) < 3e-7
    check_device_status(DEV)


@pytest.mark.parametrize("K,n,num_in,c_in,c_out", [(27, 1, 1, 64, 32), (27, 129, 90, 52, 48), (16, 4000, 6000, 36, 132), (32, 700, 700, 160, 16),
                                                   (27, 5000, 5000, 96, 64), (27, 70000, 70000, 64, 64), (27, 66000, 66000, 128, 256)])
def test_fp32_weight_gradient_on_the_tensor_cores(K, n, num_in, c_in, c_out):
    """Groups that end inside an offset and past the last, partial tiles, one range and many, column blocks: against sums
    in 64 bits (4e-7 is twice the largest error measured), closer to them than the FP32 pipes, twice the same bits."""
    from warpconvnet_b200.nn.functional import sparse_conv as sc
    g = torch.Generator(device=DEV).manual_seed(n)
    kmap = _random_map(K, n, num_in, g)
    nbr = kmap.neighbor_table(n)
    x, dy = torch.randn(num_in, c_in, generator=g, device=DEV), torch.randn(n, c_out, generator=g, device=DEV)
    want = torch.stack([x[nbr[k].clamp(min=0).long()].double().mul((nbr[k] >= 0)[:, None]).T @ dy.double() for k in range(K)])
    error = lambda y: float((y.double() - want).norm() / want.norm().clamp(min=1e-30))
    for tiled in (False, K <= 27):
        got = [sc.sparse_conv_wgrad(x, dy, kmap, n, tile_order=tiled) for _ in range(2)]
        check_device_status(DEV)
        assert torch.equal(*got) and error(got[0]) < 4e-7
    with pytest.MonkeyPatch.context() as m:
        query = sc.query_bytes
        m.setattr(sc, "query_bytes", lambda name, *a: 0 if name == "wcn_conv_wgrad_f32_workspace_bytes" else query(name, *a))
        pipes = sc.sparse_conv_wgrad(x, dy, kmap, n)
        assert n < 1000 or error(got[0]) <= error(pipes)
        for value, row in ((float("inf"), 0), (float("nan"), n // 2), (1e30, n - 1)):
            bad = dy.clone()
            bad[row, 3] = value
            want_bad = sc.sparse_conv_wgrad(x, bad, kmap, n)
            with pytest.MonkeyPatch.context() as back:
                back.setattr(sc, "query_bytes", query)
                got_bad = sc.sparse_conv_wgrad(x, bad, kmap, n)
            assert torch.equal(torch.isfinite(got_bad), torch.isfinite(want_bad))
            fine = torch.isfinite(want_bad)
            assert not fine.any() or rel_l2(got_bad[fine].cpu().numpy(), want_bad[fine].cpu().numpy()) < 1e-5
    check_device_status(DEV)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n,c", [(1, 8), (5, 24), (1023, 64), (70001, 96), (3000, 1000), (300, 7)])
def test_column_sums(dtype, n, c):
    """Fewer rows than a block takes at once, columns that do not divide a block, widths without a kernel: against 64 bits
    (fp32 sums of some hundred numbers, added in double), twice the same bits."""
    from warpconvnet_b200.nn.functional.sparse_conv import _column_sums
    x = torch.randn(n, c, generator=torch.Generator(device=DEV).manual_seed(n), device=DEV).to(dtype)
    got, want = _column_sums(x), x.double().sum(0)
    assert torch.equal(got, _column_sums(x))
    assert float((got.double() - want).abs().max()) <= 1e-6 * float(x.double().abs().sum(0).max())


@pytest.mark.parametrize("dtype,bias_dtype", [(torch.float32, torch.float32), (torch.float16, torch.float16), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("kind", ["same", "down", "up"])
def test_bias_of_a_training_layer(dtype, bias_dtype, kind):
    """The bias as part of the layer's node: forward and all gradients against the node without it and an addition; a graph of
    the bias gradient, and forward-mode tangents of the bias, go through torch as before."""
    coords = room_rows(5000)
    vox = make_voxels(coords, torch.randn(len(coords), 32, generator=torch.Generator().manual_seed(1)).to(dtype)).sort()
    torch.manual_seed(0)
    down = SparseConv3d(32, 48, 2, stride=2, bias=True).to(DEV).to(dtype)
    layer = {"same": SparseConv3d(32, 48, 3, bias=True), "down": down, "up": SparseConv3d(48, 32, 2, stride=2, bias=True, transposed=True)}[kind]
    layer = layer.to(DEV).to(dtype)
    layer.bias.data = torch.randn(layer.bias.shape, device=DEV).to(bias_dtype)
    if kind == "up":
        with torch.no_grad():
            vox, target = down(vox), vox
    call = (lambda v: layer(v, target)) if kind == "up" else layer
    outs = []
    for fused in (True, False):
        x = vox.feature_tensor.detach().clone().requires_grad_(True)
        bias = layer.bias
        if not fused:
            layer.bias = None
        y = call(vox.replace(batched_features=x)).feature_tensor
        if not fused:
            y = (y.double() + bias.double()).to(dtype)
            layer.bias = bias
        dy = torch.randn(y.shape, generator=torch.Generator(device=DEV).manual_seed(2), device=DEV).to(dtype)
        outs.append([y.detach(), *torch.autograd.grad(y, [x, layer.weight, bias], dy)])
    tol = {torch.float32: 1e-6, torch.float16: 2e-3, torch.bfloat16: 1e-2}[dtype]
    for got, want in zip(*outs):
        assert got.dtype == want.dtype and rel_l2(got.float().cpu().numpy(), want.float().cpu().numpy()) < tol
    x = vox.feature_tensor.detach().clone().requires_grad_(True)
    y = call(vox.replace(batched_features=x)).feature_tensor
    dy = torch.ones_like(y).requires_grad_(True)
    (gb,) = torch.autograd.grad(y, [layer.bias], dy, create_graph=True)
    (back,) = torch.autograd.grad(gb.sum(), [dy])
    assert torch.equal(back, torch.ones_like(back))
    check_device_status(DEV)


@pytest.mark.parametrize("n", [12000, 19000])
@pytest.mark.parametrize("where,value", [("x", float("inf")), ("x", float("nan")), ("x", 3.4e38), ("w", float("-inf")), ("w", 2.0 ** 64)])
def test_fp32_numbers_without_three_parts(n, where, value, monkeypatch):
    """Infinities, NaN and numbers whose partial products could overflow give what the FP32 pipes make of them."""
    g = torch.Generator(device=DEV).manual_seed(n)
    kmap = _random_map(27, n, n, g)
    x = torch.randn(n, 32, generator=g, device=DEV)
    w = torch.randn(27, 32, 32, generator=g, device=DEV)
    if where == "x":
        x[n // 2, 5] = value
    else:
        w[13, 7, 3] = value
    got = sparse_conv_fused(x, w, kmap, n)
    monkeypatch.setattr("warpconvnet_b200.nn.functional.sparse_conv._f32_workspace", lambda *a: (None, 0))
    want = sparse_conv_fused(x, w, kmap, n)
    check_device_status(DEV)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    fine = torch.isfinite(want)
    assert torch.equal(got[~fine & ~torch.isnan(want)], want[~fine & ~torch.isnan(want)])
    assert float((got[fine].double() - want[fine].double()).norm() / want[fine].double().norm()) < 1e-6


@pytest.mark.parametrize("n", [18944, 18945, 37889, 65536, 65537, 12 * 16384, 13 * 16384 + 129])
def test_every_unit_comes_once_whatever_their_order(n):
    """Rows in tile order are worked through dense supertiles first, the last windows of a launch together: one unit per
    multiprocessor, one more than that, small and large windows, whole and partial windows before the launch's tail.  The
    sum of a row runs over the same offsets either way, so that the results are those of the plain order bit for bit."""
    g = torch.Generator(device=DEV).manual_seed(n)
    present = torch.rand(27, n, generator=g, device=DEV) < torch.rand(n, generator=g, device=DEV) ** 3
    nbr = torch.where(present, torch.randint(0, n, (27, n), generator=g, device=DEV, dtype=torch.int32), torch.full((), -1, dtype=torch.int32, device=DEV))
    kmap = IntSearchResult.from_neighbor_table(nbr, n)
    x = torch.randn(n, 32, generator=g, device=DEV).half()
    w = (torch.randn(27, 32, 32, generator=g, device=DEV) * 0.1).half()
    got = []
    for tiled in (False, True):
        out = torch.full((n, 32), float("nan"), dtype=torch.float16, device=DEV)
        got.append(sparse_conv_fused(x, w, kmap, n, epilogue=ConvEpilogue(out=out), algo=CONV_TCGEN05, tile_order=tiled))
    check_device_status(DEV)
    want = sparse_conv_fused(x, w, kmap, n, algo=CONV_SIMT)
    assert torch.equal(*got) and rel_l2(got[0].float().cpu().numpy(), want.float().cpu().numpy()) < 2e-3


@pytest.mark.parametrize("n", [700, 19000])
@pytest.mark.parametrize("ex,ew", [(-116, 0), (-124, 0), (-140, 0), (0, -118), (-20, -100), (-64, -64), (-75, -68)])
def test_fp32_small_numbers_keep_their_bits(n, ex, ew):
    """Numbers whose third or second part would lie below bf16's range, subnormal ones, and pairs whose product is subnormal:
    layer and weight gradient as close to sums in 64 bits as the FP32 pipes, and (3e-7, 4e-7: see above) where the result
    itself is not subnormal."""
    from warpconvnet_b200.nn.functional import sparse_conv as sc
    g = torch.Generator(device=DEV).manual_seed(n)
    kmap = _random_map(27, n, n, g)
    nbr = kmap.neighbor_table(n)
    # (in two steps: 2 ** -140 times an fp32 number would be rounded before the multiplication)
    x = (torch.randn(n, 48, generator=g, device=DEV).double() * 2.0 ** ex).float()
    w = (torch.randn(27, 48, 64, generator=g, device=DEV).double() * 2.0 ** ew).float()
    dy = (torch.randn(n, 64, generator=g, device=DEV).double() * 2.0 ** ew).float()
    rows = [x[nbr[k].clamp(min=0).long()].double().mul((nbr[k] >= 0)[:, None]) for k in range(27)]
    want = sum(rows[k] @ w[k].double() for k in range(27)), torch.stack([r.T @ dy.double() for r in rows])
    error = lambda y, e: float((y.double() - e).norm() / e.norm())
    with pytest.MonkeyPatch.context() as m:
        got = sparse_conv_fused(x, w, kmap, n), sc.sparse_conv_wgrad(x, dy, kmap, n)
        query = sc.query_bytes
        m.setattr(sc, "query_bytes", lambda name, *a: 0 if "f32" in name else query(name, *a))
        pipes = sparse_conv_fused(x, w, kmap, n), sc.sparse_conv_wgrad(x, dy, kmap, n)
    check_device_status(DEV)
    for y, f, e, limit in zip(got, pipes, want, (3e-7, 4e-7)):
        assert error(y, e) <= 1.02 * error(f, e)
        assert error(y, e) < limit or ex + ew < -125


@pytest.mark.parametrize("n,c_out", [(300, 64), (5000, 144), (19000, 16), (19000, 160), (70000, 64)])
def test_fp32_special_numbers_stay_with_their_rows(n, c_out, monkeypatch):
    """A number that has no three parts changes the rows that name its row, as the FP32 pipes have them, and no bit of the
    others, however the offsets and columns of a tile are divided; in a row that no pair names it changes nothing."""
    g = torch.Generator(device=DEV).manual_seed(n)
    kmap = _random_map(27, n, n - 1, g)
    nbr = kmap.neighbor_table(n)
    x = torch.randn(n, 64, generator=g, device=DEV)
    w = torch.randn(27, 64, c_out, generator=g, device=DEV)
    clean = sparse_conv_fused(x, w, kmap, n)
    bad = x.clone()
    bad[n - 1] = float("nan")
    for row, value in ((0, float("inf")), (n // 3, float("nan")), (n // 2, -3e30), (n - 2, 6e11)):
        bad[row, row % 64] = value
    for tiled in (False, True):
        got = sparse_conv_fused(bad, w, kmap, n, tile_order=tiled)
        with monkeypatch.context() as m:
            m.setattr("warpconvnet_b200.nn.functional.sparse_conv._f32_workspace", lambda *a: (None, 0))
            want = sparse_conv_fused(bad, w, kmap, n, tile_order=tiled)
        check_device_status(DEV)
        named = torch.isin(nbr, torch.tensor([0, n // 3, n // 2, n - 2], device=DEV, dtype=nbr.dtype)).any(0)
        assert named.any() and torch.equal(got[~named], clean[~named])
        fine = torch.isfinite(want)
        assert torch.equal(got[~fine].nan_to_num(1.0), want[~fine].nan_to_num(1.0)) and (named[:, None] & fine).any()
        assert rel_l2(got[fine].cpu().numpy(), want[fine].cpu().numpy()) < 1e-6


@pytest.mark.parametrize("n,c_in,c_out", [(500, 64, 64), (9000, 36, 128), (20000, 160, 16), (70000, 64, 96)])
def test_fp32_special_numbers_stay_with_their_weights(n, c_in, c_out, monkeypatch):
    """A number that has no three parts changes the weight gradients that it belongs to, as the FP32 pipes have them, and no bit
    of the others: a row of every offset's matrix for one of X (none where no pair names it), a column for one of dY, to the
    present pairs only."""
    from warpconvnet_b200.nn.functional import sparse_conv as sc
    g = torch.Generator(device=DEV).manual_seed(n)
    kmap = _random_map(27, n, n - 1, g)
    x, dy = torch.randn(n, c_in, generator=g, device=DEV), torch.randn(n, c_out, generator=g, device=DEV)
    clean = sc.sparse_conv_wgrad(x, dy, kmap, n)
    query = sc.query_bytes
    for value in (float("inf"), float("nan"), -1e30):
        for rows, cols in (([n - 1], []), ([3], []), ([], [n // 2]), ([n // 4, n // 3], [0])):
            bad, bad_dy = x.clone(), dy.clone()
            for r in rows:
                bad[r, 5] = value
            for r in cols:
                bad_dy[r, c_out - 3] = value
            got = sc.sparse_conv_wgrad(bad, bad_dy, kmap, n, tile_order=True)
            with monkeypatch.context() as m:
                m.setattr(sc, "query_bytes", lambda name, *a: 0 if name == "wcn_conv_wgrad_f32_workspace_bytes" else query(name, *a))
                want = sc.sparse_conv_wgrad(bad, bad_dy, kmap, n)
            check_device_status(DEV)
            same = torch.ones(27, c_in, c_out, dtype=torch.bool, device=DEV)
            if rows and rows != [n - 1]:
                same[:, 5] = False
            if cols:
                same[:, :, (c_out - 3) // 4 * 4:(c_out - 3) // 4 * 4 + 4] = False
            ordered = sc.sparse_conv_wgrad(x, dy, kmap, n, tile_order=True)
            assert torch.equal(got[same], ordered[same]) and rel_l2(ordered.cpu().numpy(), clean.cpu().numpy()) < 1e-6
            fine = torch.isfinite(want)
            assert torch.equal(got[~fine].nan_to_num(1.0), want[~fine].nan_to_num(1.0))
            fine &= ~same
            # (sums of N = n / 3 products one after the other: N roundings of 2^-24 of partial sums that grow as their square
            # root, 2^-25 (N / 6)^1/2 = 2e-6 of the total for the longest, on both sides)
            assert not fine.any() or rel_l2(got[fine].cpu().numpy(), want[fine].cpu().numpy()) < 1e-5


@pytest.mark.parametrize("c_in,c_out", [(32, 32), (64, 64), (36, 36), (128, 144)])
def test_fp32_rows_do_not_depend_on_their_launch(c_in, c_out):
    """What a scene divided among GPUs relies on (interior rows, boundary rows, all rows at once; halo rows that have not
    arrived yet hold anything): with ``split_k=1`` a row's bits are those of the launch over all rows."""
    g = torch.Generator(device=DEV).manual_seed(c_in)
    n = 45000
    kmap = _random_map(27, n, n, g)
    nbr = kmap.neighbor_table(n)
    x = torch.randn(n + 50, c_in, generator=g, device=DEV)
    w = torch.randn(27, c_in, c_out, generator=g, device=DEV)
    whole = sparse_conv_fused(x, w, kmap, n, split_k=1)
    x[n:] = float("nan")
    for rows in (slice(0, 90), slice(17000, 18000), slice(5000, 45000)):
        part = IntSearchResult.from_neighbor_table(nbr[:, rows].contiguous(), n + 50)
        got = sparse_conv_fused(x, w, part, len(range(n)[rows]), split_k=1)
        check_device_status(DEV)
        assert torch.equal(got, whole[rows])


def _fastest(f):
    times = []
    for _ in range(9):
        torch.cuda._sleep(400000)   # (the launches are there before the first one starts)
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        f()
        end.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(end))
    return sorted(times)[2]


@pytest.mark.parametrize("n,c_out", [(300, 176), (19000, 208), (2000, 272), (20000, 400)])
def test_fp32_column_blocks_of_different_widths(n, c_out):
    """Widths above 128 columns that equal blocks of sixteens do not divide well, with offsets divided among a cluster and not:
    against sums in 64 bits, forward and weight gradient (the bounds above)."""
    from warpconvnet_b200.nn.functional import sparse_conv as sc
    g = torch.Generator(device=DEV).manual_seed(c_out)
    kmap = _random_map(27, n, n, g)
    nbr = kmap.neighbor_table(n)
    x, dy = torch.randn(n, 48, generator=g, device=DEV), torch.randn(n, c_out - 12, generator=g, device=DEV)
    w = torch.randn(27, 48, c_out, generator=g, device=DEV)
    rows = [x[nbr[k].clamp(min=0).long()].double().mul((nbr[k] >= 0)[:, None]) for k in range(27)]
    want = sum(rows[k] @ w[k].double() for k in range(27)), torch.stack([r.T @ dy.double() for r in rows])
    got = sparse_conv_fused(x, w, kmap, n), sc.sparse_conv_wgrad(x, dy, kmap, n)
    check_device_status(DEV)
    for y, e, limit in zip(got, want, (3e-7, 4e-7)):
        assert float((y.double() - e).norm() / e.norm()) < limit


def test_fp32_column_blocks_are_few():
    """A layer gathers its rows once per column block: 208 columns take two blocks, not thirteen of sixteen, and a gradient of
    160 two, not five (5.1 and 3.3 times a layer of 112 and a gradient of 80 columns before, 1.6 and 1.7 times with two)."""
    from warpconvnet_b200.nn.functional import sparse_conv as sc
    g = torch.Generator(device=DEV).manual_seed(0)
    n = 40000
    kmap = _random_map(27, n, n, g)
    x = torch.randn(n, 64, generator=g, device=DEV)
    layer = lambda c: _fastest(lambda w=torch.randn(27, 64, c, generator=g, device=DEV): sparse_conv_fused(x, w, kmap, n))
    grad = lambda c: _fastest(lambda dy=torch.randn(n, c, generator=g, device=DEV): sc.sparse_conv_wgrad(x, dy, kmap, n))
    ratio = layer(208) / layer(112), grad(160) / grad(80)
    assert ratio[0] < 3 and ratio[1] < 2.6
    check_device_status(DEV)


@pytest.mark.parametrize("n,c", [(300000, 1024), (800000, 256), (1000000, 16)])
def test_column_sums_of_many_rows(n, c):
    """A thread adds hundreds to thousands of rows of these.  Trees of eight numbers in fp32 (three additions deep, each half a
    unit of 2^-24 off at most) and a result rounded once, everything else in double: below 1e-7 of the sums' 2-norm."""
    from warpconvnet_b200.nn.functional.sparse_conv import _column_sums
    x = torch.randn(n, c, generator=torch.Generator(device=DEV).manual_seed(c), device=DEV)
    want = x.sum(0, dtype=torch.float64)
    assert float((_column_sums(x).double() - want).norm() / want.norm()) < 1e-7


@pytest.mark.parametrize("frozen", [True, False])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_gradient_of_a_bias_alone(dtype, frozen):
    """A layer of which only the bias trains keeps nothing for the backward pass; the gradient of a bias alone does not run the
    layer's, one by one, in batches (``is_grads_batched``) and, as a tangent, in forward mode."""
    import torch.autograd.forward_ad as fwd
    from warpconvnet_b200._native import LAUNCH_COUNTS
    coords = room_rows(3000)
    vox = make_voxels(coords, torch.randn(len(coords), 32, generator=torch.Generator().manual_seed(1)).to(dtype)).sort()
    torch.manual_seed(0)
    layer = SparseConv3d(32, 48, 3, bias=True).to(DEV).to(dtype)
    layer.weight.requires_grad_(not frozen)
    kept = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (kept.append(t), t)[1], lambda t: t):
        y = layer(vox).feature_tensor
    assert type(y.grad_fn).__name__ == "_BiasFunctionBackward" and len(kept) == (0 if frozen else 2)
    dys = torch.randn(3, *y.shape, generator=torch.Generator(device=DEV).manual_seed(2), device=DEV).to(dtype)
    want = dys.double().sum(1)
    close = lambda a, b: rel_l2(a.double().cpu().numpy(), b.cpu().numpy()) < (1e-6 if dtype == torch.float32 else 1e-3)
    LAUNCH_COUNTS.clear()
    for dy, w in zip(dys, want):
        assert close(torch.autograd.grad(y, [layer.bias], dy, retain_graph=True)[0], w)
    assert LAUNCH_COUNTS["wcn_column_sums"] == 3 * 2 and not any(c for k, c in LAUNCH_COUNTS.items() if "conv" in k)
    assert close(torch.autograd.grad(y, [layer.bias], dys, is_grads_batched=True)[0], want)
    if frozen:  # (without a parameter that trains a call is one of inference)
        return
    with fwd.dual_level():
        bias = layer.bias
        del layer.bias
        layer.bias = fwd.make_dual(bias.detach(), torch.full_like(bias.detach(), 0.5))
        tangent = fwd.unpack_dual(layer(vox).feature_tensor).tangent
        assert tangent is not None and torch.equal(tangent, torch.full_like(y, 0.5))
    check_device_status(DEV)


def test_fp32_launches_are_counted():
    """Planes and convolution are two kernels, the FP32 pipes one; the weight gradient has a third where there are partial sums."""
    from warpconvnet_b200._native import LAUNCH_COUNTS
    from warpconvnet_b200.nn.functional import sparse_conv as sc
    g = torch.Generator(device=DEV).manual_seed(0)

    def counted(n, c, name, f):
        kmap = _random_map(27, n, n, g)
        kmap.tile_masks(n)
        x, y, w = (torch.randn(*shape, generator=g, device=DEV) for shape in ((n, c), (n, c), (27, c, c)))
        LAUNCH_COUNTS.clear()
        f(x, y, w, kmap, n)
        return LAUNCH_COUNTS[name]

    forward, gradient = lambda x, y, w, kmap, n: sparse_conv_fused(x, w, kmap, n), lambda x, y, w, kmap, n: sc.sparse_conv_wgrad(x, y, kmap, n)
    assert counted(3000, 64, "wcn_conv_fwd", forward) == 2 and counted(3000, 36, "wcn_conv_fwd", forward) == 1
    assert counted(400, 64, "wcn_conv_wgrad_f32", gradient) == 2 and counted(20000, 64, "wcn_conv_wgrad_f32", gradient) == 3
    check_device_status(DEV)


def test_fp32_kernels_are_loud_after_an_expired_wait():
    """While the status word holds an expired wait the fp32 kernels write NaN, sums that are made again among them."""
    from warpconvnet_b200._native import device_status, lib, ptr, stream_ptr
    from warpconvnet_b200.nn.functional import sparse_conv as sc
    g = torch.Generator(device=DEV).manual_seed(0)
    n, dev = 6000, torch.device(DEV)
    kmap = _random_map(27, n, n, g)
    x, dy, w = (torch.randn(*shape, generator=g, device=DEV) for shape in ((n, 64), (n, 64), (27, 64, 64)))
    calls = [lambda s=s: sparse_conv_fused(x, w, kmap, n, split_k=s) for s in (1, 4)] + [lambda: sc.sparse_conv_wgrad(x, dy, kmap, n)]
    x[5, 5] = float("inf")
    right = [f() for f in calls]
    check_device_status(DEV)
    assert lib().wcn_selftest_bounded_wait(200_000, ptr(device_status(dev)), None, stream_ptr(dev)) == 0
    loud = [f() for f in calls]
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="expired"):
        check_device_status(DEV)
    assert all(bool(torch.isnan(y).all()) for y in loud)
    assert all(torch.equal(a.nan_to_num(1.0), f().nan_to_num(1.0)) for a, f in zip(right, calls))
    check_device_status(DEV)


def test_gradients_of_an_input_and_a_bias_in_parts():
    """Whichever of a layer's three gradients are asked for, together or one by one, they have the same bits, behind an input that is a
    leaf and one that is not; batches of bias gradients do not run the layer's either way."""
    coords = room_rows(3000)
    vox = make_voxels(coords, torch.randn(len(coords), 64, generator=torch.Generator().manual_seed(1))).sort()
    torch.manual_seed(0)
    layer = SparseConv3d(64, 48, 3, bias=True).to(DEV)
    x = vox.feature_tensor.detach().clone().requires_grad_(True)
    for feats in (x, x * 1.0):
        y = layer(vox.replace(batched_features=feats)).feature_tensor
        dy = torch.randn(y.shape, generator=torch.Generator(device=DEV).manual_seed(2), device=DEV)
        asked = {"x": x, "w": layer.weight, "b": layer.bias}
        want = dict(zip(asked, torch.autograd.grad(y, list(asked.values()), dy, retain_graph=True)))
        for names in ("x", "w", "b", "xw", "xb", "wb"):
            got = torch.autograd.grad(y, [asked[k] for k in names], dy, retain_graph=True)
            assert all(torch.equal(a, want[k]) for a, k in zip(got, names))
        batch = torch.stack([dy, -dy])
        (gb,) = torch.autograd.grad(y, [layer.bias], batch, retain_graph=True, is_grads_batched=True)
        assert rel_l2(gb[0].cpu().numpy(), want["b"].cpu().numpy()) < 1e-6 and torch.equal(gb[0], -gb[1])
        y.backward(dy, inputs=[layer.bias])
        assert torch.equal(layer.bias.grad, want["b"]) and layer.weight.grad is None and x.grad is None
        layer.bias.grad = None
    check_device_status(DEV)
