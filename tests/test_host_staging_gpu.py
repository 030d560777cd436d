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


# (64 KB are 16 rows of 1024 columns, 128 KB 31 with two slots each, 256 KB 64)
@pytest.mark.parametrize("T", [1, 16, 17, 31, 32, 63, 64, 200, 256])
@pytest.mark.parametrize("locked_in,locked_out", [(True, True), (True, False), (False, True)])
@pytest.mark.parametrize("mixed", [False, True])
def test_page_locked_buffers(gpu_lib, T, locked_in, locked_out, mixed):
    """Page-locked buffers are copied without staging (small results with it), in any mixture: the same results, and nothing written
    by a call that fails."""
    sh = synth.tiny(seed=70 + T, E=8, k=2, H=1024, F=64, T=T, has_bias=True)
    h, Wg, rb, ex = cases.layer_inputs(sh)
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    out, ro = np.full((T, 1024), 7, np.float32), np.full((T, 2, 2), 7, np.float32)
    lay.forward(h, out=out, router_out_buf=ro)

    def host(shape, locked):
        return torch.full(shape, 5.0, pin_memory=locked).numpy()

    # mixed: the routing is in the other kind of memory than the rows
    x, x_route = host((T, 1024), locked_in), host((T, 2, 2), locked_in != mixed)
    got, got_ro = host((T, 1024), locked_out), host((T, 2, 2), locked_out != mixed)
    x[:], x_route[:] = h, ro
    for given in (None, x_route):
        for _ in range(2):
            got[:], got_ro[:] = 5, 5
            lay.forward(x, router_out=given, out=got, router_out_buf=got_ro)
            assert np.array_equal(got, out) and np.array_equal(got_ro, ro)
    x_route[T - 1, 1, 0] = 8
    with pytest.raises(CskError, match="out of range"):
        lay.forward(x, router_out=x_route, out=got, router_out_buf=got_ro)
    assert np.array_equal(got, out) and np.array_equal(got_ro, ro)
    lay.close()


@pytest.mark.parametrize("T", [95, 96])  # 384 KB of results and routing are 95 rows
def test_page_locked_results_at_the_line(gpu_lib, T):
    test_page_locked_buffers(gpu_lib, T, True, True, False)


@pytest.mark.parametrize("T", [900, 2000])  # more tokens than six an SM, in results that still fit the staging area
def test_short_rows_of_many_tokens(gpu_lib, T):
    sh = synth.tiny(seed=T, E=8, k=2, H=64, F=64, T=T, has_bias=True)
    h, Wg, rb, ex = cases.layer_inputs(sh)
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    out, ro = np.full((T, 64), 7, np.float32), np.full((T, 2, 2), 7, np.float32)
    x, got, got_ro = torch.from_numpy(h).cuda(), torch.empty((T, 64), device="cuda"), torch.empty((T, 2, 2), device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        out[:], ro[:] = 7, 7
        lay.forward(h, out=out, router_out_buf=ro)
        lay.forward_dev(x, T, got, d_router_out=got_ro)
        lay.sync()
        assert np.array_equal(out, got.cpu().numpy()) and np.array_equal(ro, got_ro.cpu().numpy())
    lay.close()
