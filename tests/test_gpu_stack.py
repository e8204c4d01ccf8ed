"""``nn.SparseUNet`` as one autograd node against its layers one by one: outputs and gradients, whichever inputs need one; what
makes it run layer by layer; and the two small kernels behind it, at sizes that fill no vector and no block."""
import contextlib
import ctypes
import gc

import pytest
import torch

from fgms_b200 import _lib, clouds, nn, unet

pytestmark = pytest.mark.gpu

SPEC = unet.minkunet_spec(4, (16, 32, 48))


def _net(spec=SPEC, dtype=torch.float16, n=3000, side=20):
    coords = torch.from_numpy(clouds.uniform_cloud(n, side, 7)).cuda()
    umaps = unet.build_unet_maps(coords, (len(spec) - 1) // 6)
    torch.manual_seed(3)
    net = nn.SparseUNet(spec, dtype=dtype)
    with torch.no_grad():
        for layer in net.layers:
            layer.weight.mul_(2.0)
    feats = torch.randn((coords.size(0), spec[0].c_in), device="cuda").to(dtype)
    grad = torch.randn((coords.size(0), spec[-1].c_out), device="cuda").to(dtype)
    return net, umaps, feats, grad


def _layer_by_layer(net, feats, umaps):
    val = {"input": feats}
    for spec, layer in zip(net.spec, net.layers):
        y = layer(val[spec.src], umaps.of(spec))
        val[spec.dst] = y if spec.skip is None else y + val[spec.skip]
    return val[net.spec[-1].dst]


def _close(a, b, dtype):
    # the same sums in another order: at most 27 (forward, input gradient) or a few hundred partial sums, through 13 layers
    tol = 2e-2 if dtype == torch.float16 else 1e-2
    assert float((a.double() - b.double()).norm()) <= tol * float(b.double().norm())


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("needs", ["all", "weights", "input", "last", "frozen_middle", "first"])
def test_one_node_equals_a_node_per_layer(dtype, needs):
    net, umaps, feats, grad = _net(dtype=dtype)
    params = list(net.parameters())
    for i, p in enumerate(params):
        p.requires_grad_({"all": True, "weights": True, "input": False, "last": i == len(params) - 1,
                          "frozen_middle": i % 3 != 1, "first": i == 0}[needs])
    feats.requires_grad_(needs in ("all", "input", "frozen_middle"))
    wanted = [t for t in [feats] + params if t.requires_grad]
    got, want = net(feats, umaps), _layer_by_layer(net, feats, umaps)
    assert got.grad_fn.name() != want.grad_fn.name()
    _close(got.detach(), want.detach(), dtype)
    for a, b in zip(torch.autograd.grad(got, wanted, grad, retain_graph=True), torch.autograd.grad(want, wanted, grad)):
        _close(a, b, dtype)
    for a, b in zip(torch.autograd.grad(got, wanted[-1:], grad), wanted[-1:]):  # a second backward, of one of them
        assert a.shape == b.shape


NEEDS = ["all", "weights", "input", "last", "frozen_middle", "first"]


def _compare(net, umaps, feats, grad, needs):
    params, dtype = list(net.parameters()), feats.dtype
    for i, p in enumerate(params):
        p.requires_grad_({"all": True, "weights": True, "input": False, "last": i == len(params) - 1,
                          "frozen_middle": i % 3 != 1, "first": i == 0}[needs])
    feats.requires_grad_(needs in ("all", "input", "frozen_middle"))
    wanted = [t for t in [feats] + params if t.requires_grad]
    got, want = net(feats, umaps), _layer_by_layer(net, feats, umaps)
    assert got.grad_fn.name() != want.grad_fn.name()
    _close(got.detach(), want.detach(), dtype)
    first, second = torch.autograd.grad(got, wanted, grad, retain_graph=True), torch.autograd.grad(want, wanted, grad)
    for a, b in zip(first, second):
        _close(a, b, dtype)
    # further backwards, of some of them: a layer in the middle, the last one, and the first and the last
    middle = len(wanted) // 2
    for some in ([middle], [len(wanted) - 1], [0, len(wanted) - 1]):
        again = torch.autograd.grad(got, [wanted[i] for i in some], grad, retain_graph=some != [0, len(wanted) - 1])
        for i, a in zip(some, again):
            _close(a, second[i], dtype)
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(got, wanted[-1:], grad)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("needs", NEEDS)
def test_further_backwards_over_a_retained_graph(dtype, needs):
    _compare(*_net(dtype=dtype), needs)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("needs", NEEDS)
def test_values_and_gradients_one_by_one(dtype, needs):
    """120 MB of values, 240 in fp32: more than are held in one allocation."""
    _compare(*_net(dtype=dtype, n=240000, side=160), needs)


@contextlib.contextmanager
def _no_more_than(extra):
    """Of the memory that is reserved nothing is left that 1 MB fit in, and `extra` bytes can be reserved beyond it."""
    gc.collect()  # what earlier tests left in cycles would otherwise be handed back at any time
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    limit, held = torch.cuda.get_device_properties(0).total_memory, []
    try:
        torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / limit)
        for size in [1 << k for k in range(28, 19, -1)]:
            with contextlib.suppress(torch.OutOfMemoryError):
                while True:
                    held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + extra) / limit)
        yield
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


def _in_64_bits(net, umaps, feats, grad, wanted):
    """The same layers in plain PyTorch, fp64: output and gradients."""
    twin = {t: t.detach().double().requires_grad_() for t in wanted}
    val = {"input": twin.get(feats, feats.double())}
    for spec, layer in zip(net.spec, net.layers):
        km, x, w = umaps.of(spec), val[spec.src], twin.get(layer.weight, layer.weight.detach().double())
        at, im, om = km.kpos.tolist(), km.imap.long(), km.omap.long()
        y = torch.zeros((km.n_out, w.size(2)), dtype=torch.double, device="cuda")
        for k in range(w.size(0)):
            y = y.index_add(0, om[at[k]:at[k + 1]], x[im[at[k]:at[k + 1]]] @ w[k])
        val[spec.dst] = y if spec.skip is None else y + val[spec.skip]
    out = val[net.spec[-1].dst]
    return out.detach(), torch.autograd.grad(out, [twin[t] for t in wanted], grad.double())


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_against_64_bits(dtype):
    # a layer rounds its inputs (tf32) or up to ten partial sums of a row (fp16) to 11 bits: 1e-3 relative at most, and 13 layers
    # there and 13 back in quadrature 5e-3; the bound is _close's
    net, umaps, feats, grad = _net(dtype=dtype)
    feats.requires_grad_()
    wanted = [feats] + list(net.parameters())
    got = net(feats, umaps)
    out, grads = _in_64_bits(net, umaps, feats, grad, wanted)
    _close(got.detach(), out, dtype)
    for a, b in zip(torch.autograd.grad(got, wanted, grad), grads):
        _close(a, b, dtype)


def test_layers_of_a_million_pairs():
    """The finest layers take the kernel for both gradients, with a workspace."""
    net, umaps, feats, grad = _net(n=60000, side=40)
    assert umaps.subm[0].imap.numel() > 1 << 20
    feats.requires_grad_()
    wanted = [feats] + list(net.parameters())
    got, want = net(feats, umaps), _layer_by_layer(net, feats, umaps)
    _close(got.detach(), want.detach(), torch.float16)
    for a, b in zip(torch.autograd.grad(got, wanted, grad), torch.autograd.grad(want, wanted, grad)):
        _close(a, b, torch.float16)


@pytest.mark.parametrize("n,side", [(3000, 20), (240000, 160)])  # two allocations, and one by one
def test_on_another_stream_and_in_a_captured_graph(n, side):
    net, umaps, feats, grad = _net(n=n, side=side)
    params = list(net.parameters())

    def step():
        out = net(feats, umaps)
        return (out.detach(), *torch.autograd.grad(out, params, grad))

    want, stream = step(), torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for a, b in zip(step(), want):
            _close(a, b, torch.float16)
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step()
    for t in got:
        t.fill_(float("nan"))
    for _ in range(2):
        graph.replay()
    for a, b in zip(got, want):
        _close(a, b, torch.float16)


def test_a_step_takes_no_more_memory_than_a_node_per_layer():
    net, umaps, feats, grad = _net(n=240000, side=160)
    params = list(net.parameters())

    def peak(forward):
        torch.autograd.grad(forward(), params, grad)
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        torch.autograd.grad(forward(), params, grad)
        return torch.cuda.max_memory_allocated() - before

    assert peak(lambda: net(feats, umaps)) <= 1.02 * peak(lambda: _layer_by_layer(net, feats, umaps))


def test_without_memory_for_all_gradients_at_once():
    """Of 100 k voxels all values' gradients are 50 MB, those in use at a time 16."""
    net, umaps, feats, grad = _net(n=100000, side=120)
    feats.requires_grad_()
    wanted = [feats] + list(net.parameters())
    out = net(feats, umaps)
    want = torch.autograd.grad(out, wanted, grad, retain_graph=True)
    with _no_more_than(40 << 20):
        with pytest.raises(torch.OutOfMemoryError):
            torch.empty(48 << 20, dtype=torch.uint8, device="cuda")
        got = torch.autograd.grad(out, wanted, grad)
    for a, b in zip(got, want):
        _close(a, b, torch.float16)


def test_without_memory_for_all_values_at_once():
    """200 MB are free, but in pieces of 18 MB (beyond them 16 for small tensors)."""
    net, umaps, feats, grad = _net(n=100000, side=120)
    params = list(net.parameters())
    want = torch.autograd.grad(net(feats, umaps), params, grad)
    with _no_more_than(236 << 20):
        pieces = [torch.empty(2 << 20, dtype=torch.uint8, device="cuda") for _ in range(110)]
        kept = pieces[::10]
        del pieces
        with pytest.raises(torch.OutOfMemoryError):
            torch.empty(24 << 20, dtype=torch.uint8, device="cuda")
        out = net(feats, umaps)
        assert "Stack" in out.grad_fn.name()
        got = torch.autograd.grad(out, params, grad)
    assert len(kept) == 11
    for a, b in zip(got, want):
        _close(a, b, torch.float16)


def test_no_gradients_and_in_place_changes():
    net, umaps, feats, grad = _net()
    with torch.no_grad():
        assert not net(feats, umaps).requires_grad
    out = net(feats, umaps)
    with torch.no_grad():
        net.layers[2].weight.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.backward(grad)


def test_what_sees_the_layers_has_them_run_one_by_one():
    net, umaps, feats, grad = _net()
    one = net(feats, umaps).grad_fn.name()
    calls = []
    handle = net.layers[1].register_forward_hook(lambda *a: calls.append(1))
    assert net(feats, umaps).grad_fn.name() != one and calls == [1]
    handle.remove()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t):
        assert net(feats, umaps).grad_fn.name() != one
    assert net(feats, umaps).grad_fn.name() == one
    assert net(feats.t().contiguous().t(), umaps).grad_fn.name() != one  # layer by layer takes any strides
    with pytest.raises(ValueError):
        net(feats[:-1].contiguous(), umaps)
    with pytest.raises(ValueError):
        net(feats.float(), umaps)


def test_a_value_that_two_layers_read_has_a_node_per_layer():
    spec = [unet.LayerSpec("a", "subm", 16, 16, 0, 0, "input", "x"), unet.LayerSpec("b", "subm", 16, 16, 0, 0, "x", "y"),
            unet.LayerSpec("c", "subm", 16, 16, 0, 0, "x", "z", skip="y")]
    coords = torch.from_numpy(clouds.uniform_cloud(500, 12, 7)).cuda()
    umaps, net = unet.build_unet_maps(coords, 1), nn.SparseUNet(spec)
    feats = torch.randn((coords.size(0), 16), device="cuda").half()
    assert net._forward_as_one(feats, umaps) is None
    net(feats, umaps).sum().backward()
    assert all(float(p.grad.abs().max()) > 0 for p in net.parameters())


@pytest.mark.parametrize("sizes", [[1], [15, 16, 17], [16384, 16385, 0, 3], [7] * 70 + [40000], [1 << 22]])
def test_zero_list(sizes):
    buffers = [torch.full((n + 16,), 7, dtype=torch.uint8, device="cuda") for n in sizes]
    at = (ctypes.c_void_p * len(sizes))(*[b.data_ptr() for b in buffers])
    _lib.check(_lib.lib.fgms_b200_zero_list(at, (ctypes.c_size_t * len(sizes))(*sizes), len(sizes), torch.cuda.current_stream().cuda_stream))
    for b, n in zip(buffers, sizes):
        assert not b[:n].any() and bool((b[n:] == 7).all())


@pytest.mark.parametrize("count", [1, 3, 8, 9, 4095, 65537, 3000001])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_add(count, dtype):
    y, x = torch.randn(count + 8, device="cuda").to(dtype), torch.randn(count + 8, device="cuda").to(dtype)
    want = torch.cat([y[:count] + x[:count], y[count:]])
    _lib.check(_lib.lib.fgms_b200_add(y.data_ptr(), x.data_ptr(), count, 1 if dtype == torch.float16 else 0, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(y, want)


@pytest.mark.parametrize("c_in", [1, 5, 17, 30])
def test_input_channels_that_are_padded(c_in):
    net, umaps, feats, grad = _net(unet.minkunet_spec(c_in, (16, 32, 48)))
    feats.requires_grad_()
    wanted = [feats] + list(net.parameters())
    got, want = net(feats, umaps), _layer_by_layer(net, feats, umaps)
    _close(got.detach(), want.detach(), torch.float16)
    for a, b in zip(torch.autograd.grad(got, wanted, grad), torch.autograd.grad(want, wanted, grad)):
        assert a.is_contiguous()
        _close(a, b, torch.float16)


@pytest.mark.parametrize("rows,length,src_pitch,dst_pitch", [(1, 1, 1, 1), (257, 3, 5, 16), (27, 128, 128, 512), (100003, 4, 4, 16)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_copy_rows(rows, length, src_pitch, dst_pitch, dtype):
    src, dst = torch.randn((rows, src_pitch), device="cuda").to(dtype), torch.full((rows, dst_pitch), 7.0, device="cuda").half()
    want = dst.clone()
    want[:, :length] = src[:, :length].half()
    _lib.check(_lib.lib.fgms_b200_copy_rows_f16(src.data_ptr(), src_pitch, 1 if dtype == torch.float16 else 0, dst.data_ptr(), dst_pitch, rows, length,
                                                torch.cuda.current_stream().cuda_stream))
    assert torch.equal(dst, want)
