"""A host thread whose first CUDA call is one of the tcgen05 kernels', after another thread has used the same shape: the C ABI
needs nothing of a thread beyond a current device."""
import threading

import pytest
import torch

from fgms_b200 import _lib, clouds, maps
from tests.util import Problem

pytestmark = pytest.mark.gpu


def test_first_call_of_a_thread():
    from fgms_b200 import backend
    L, f16, m16 = _lib.lib, _lib.DTYPE_F16, _lib.MATH_F16
    p = Problem(maps.build_submanifold_map(clouds.uniform_cloud(700, 12, seed=3), 3), 128, 128, seed=1, mode="fp16")
    n, pairs, k_vol = p.km.n_in, p.km.pairs, p.km.k_vol
    table = backend.build_neighbor_table(p.kpos, p.imap, p.omap, n, n)
    feats, weights, grad, kpos, imap, omap, nbr = (t.data_ptr() for t in (p.feats, p.weights, p.grad_out, p.kpos, p.imap, p.omap, table))
    passes = [
        lambda out: L.fgms_b200_fusion_fwd(feats, weights, out, kpos, None, imap, omap, pairs, n, n, 128, 128, 128, k_vol, 0, f16, m16, 0, None),
        lambda out: L.fgms_b200_dgrad(grad, weights, out, kpos, imap, omap, pairs, n, n, 128, 128, k_vol, f16, m16, None),
        lambda out: L.fgms_b200_fwd_output_stationary(feats, weights, out, nbr, n, n, 128, 128, k_vol, f16, m16, None, 0, 0, None),
    ]
    mine, theirs = (torch.zeros((3, n, 128), dtype=torch.float16, device="cuda") for _ in range(2))
    for i, call in enumerate(passes):
        assert call(mine[i].data_ptr()) == 0, _lib.last_error()
    torch.cuda.synchronize()
    to, said = [theirs[i].data_ptr() for i in range(3)], []
    for call, out in zip(passes, to):
        t = threading.Thread(target=lambda: said.append((call(out), _lib.last_error())))
        t.start()
        t.join()
    assert [rc for rc, _ in said] == [0, 0, 0], said
    torch.cuda.synchronize()
    assert torch.allclose(mine.float(), theirs.float(), rtol=0, atol=float(mine.float().abs().max()) * 1e-2)  # reds in another order, fp16
