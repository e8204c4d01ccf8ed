"""What ``nn.SparseUNet`` hands to the node for a whole stack (no GPU: the node's entry point is a stand-in that records it)."""
import types

import pytest
import torch

from fgms_b200 import nn, unet

SPEC = unet.minkunet_spec(4, (16, 32, 48))


class _MapsPerCall:
    """Kernel maps whose objects are made for every question: only what is kept of one lives on."""

    def of(self, layer):
        name = (layer.kind, min(layer.res_in, layer.res_out))
        code = 100 * ("subm", "down", "up").index(layer.kind) + name[1]
        tensors = [torch.full((1,), code, dtype=torch.int32) for _ in range(3)]
        return types.SimpleNamespace(kpos=tensors[0], imap=tensors[1], omap=tensors[2], n_in=code, n_out=code + 1)


@pytest.fixture
def handed(monkeypatch):
    got = []
    monkeypatch.setattr(nn, "_native", types.SimpleNamespace(sparse_stack=lambda *a: got.append(a) or a[0]))
    return got


def test_every_layer_gets_its_own_map(handed):
    net, maps = nn.SparseUNet(SPEC, device="cpu"), _MapsPerCall()
    net(torch.zeros((2, 4), dtype=torch.float16), maps)
    (_, weights, tensors, plan, _), = handed
    assert len(weights) == len(SPEC) and len(plan) == 5 * len(SPEC)
    for i, layer in enumerate(SPEC):
        want, (m, n_in, n_out) = maps.of(layer), plan[5 * i + 2: 5 * i + 5]
        assert [int(t) for t in tensors[3 * m: 3 * m + 3]] == [want.n_in] * 3 and (n_in, n_out) == (want.n_in, want.n_out)


@pytest.mark.parametrize("owner,name", [(torch._C, "_get_tracing_state"), (torch.autograd.forward_ad, "_current_level"),
                                        (torch._C._functorch, "peek_interpreter_stack"), (torch._C._autograd, "_top_saved_tensors_default_hooks"),
                                        (torch._C, "_len_torch_function_stack"), (torch.nn.modules.module, "_global_forward_hooks")])
def test_a_release_without_a_private_name_runs_layer_by_layer(handed, monkeypatch, owner, name):
    net, feats = nn.SparseUNet(SPEC, device="cpu"), torch.zeros((2, 4), dtype=torch.float16)
    with monkeypatch.context() as m:
        m.delattr(owner, name)
        one = net._forward_as_one(feats, _MapsPerCall())
    assert one is None and not handed
    assert net._forward_as_one(feats, _MapsPerCall()) is feats
