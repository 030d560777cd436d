"""Host buffers around the size up to which they go through the handle's own staging: the device entry's results bit for bit, the
caller's routing or the router's, and nothing written by a call that fails."""
import numpy as np
import pytest
import torch

from coalsack_b200 import CskError, MoeLayer, synth
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 2, 3, 255, 256])  # 1 MB each way are 255 rows of 1024 columns with two slots
@pytest.mark.parametrize("routed", [True, False])
def test_results_and_errors(gpu_lib, T, routed):
    sh = synth.tiny(seed=90 + T, E=8, k=2, H=1024, F=64, T=T, has_bias=True)
    h, Wg, rb, ex = cases.layer_inputs(sh)
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    rng = np.random.default_rng(T)
    route = rng.uniform(0.1, 1.0, (T, 2, 2)).astype(np.float32)
    route[..., 0] = [rng.permutation(8)[:2] for _ in range(T)]
    given = None if routed else route
    out, ro = np.full((T, 1024), 7, np.float32), np.full((T, 2, 2), 7, np.float32)
    for _ in range(2):
        lay.forward(h, router_out=given, out=out, router_out_buf=ro)
    x, got, got_ro = torch.from_numpy(h).cuda(), torch.empty((T, 1024), device="cuda"), torch.empty((T, 2, 2), device="cuda")
    r = None if routed else torch.from_numpy(route).cuda()
    torch.cuda.synchronize()
    lay.forward_dev(x, T, got, d_router_in=r, d_router_out=got_ro)
    lay.sync()
    assert np.array_equal(out, got.cpu().numpy()) and np.array_equal(ro, got_ro.cpu().numpy())
    bad = route.copy()
    bad[0, 0, 0] = 8
    kept_out, kept_ro = out.copy(), ro.copy()
    with pytest.raises(CskError, match="out of range"):
        lay.forward(h, router_out=bad, out=out, router_out_buf=ro)
    assert np.array_equal(out, kept_out) and np.array_equal(ro, kept_ro)
    lay.forward(h, router_out=given, out=out, router_out_buf=ro)
    assert np.array_equal(out, kept_out) and np.array_equal(ro, kept_ro)
    lay.close()
