"""How many passes the host entry point cuts a batch into, by the memory of its buffers and the work that a pass would have.

The last pass's launches tell its size: up to 8192 (token, expert) pairs are planned by one launch, more by two."""
import numpy as np
import pytest
import torch

from coalsack_b200 import CskError, MoeLayer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,F,T,f16,pinned,most", [
    (64, 64, 12800, False, False, 12800),  # pageable, 200 rows per expert: one pass
    (64, 64, 12800, False, True, 6400),    # page-locked: two
    (32, 256, 20000, False, False, 10000),  # pageable, 625: two
    (32, 256, 20000, False, True, 4000),   # page-locked: five
    (80, 64, 20000, False, True, 10000),   # 250 rows, copies of 5 MB: still two ...
    (96, 64, 24500, False, True, 8167),    # ... and of 6.3 MB: three
    (1, 64, 20000, True, True, 10000),     # one expert without work for more than two
])
def test_passes(gpu_lib, E, F, T, f16, pinned, most):
    H = 64
    rng = np.random.default_rng(E)
    lay = MoeLayer(E, 1, H, F, activation=1, has_bias=False, max_tokens=T, weights_f16=f16)
    for e in range(E):
        if f16:
            lay.load_expert_f16(e, *((rng.standard_normal(s) * 0.1).astype(np.float16) for s in ((F, H), (F, H), (H, F))))
        else:
            b = [np.full((F * H // 32, 17), 120, np.uint8) for _ in range(3)]
            for m in b:
                m[:, 1:] = rng.integers(0, 256, m[:, 1:].shape)
            lay.load_expert(e, *(m.reshape(-1) for m in b))
    hidden = torch.from_numpy(rng.standard_normal((T, H)).astype(np.float32))
    route = torch.ones(T, 1, 2)
    route[:, 0, 0] = torch.arange(T) % E
    out = torch.empty(T, H)
    if pinned:
        hidden, route, out = hidden.pin_memory(), route.pin_memory(), out.pin_memory()

    def launches(n):
        lay.forward_dev(hidden[:n].cuda(), n, torch.empty(n, H, device="cuda"), d_router_in=route[:n].cuda())
        lay.sync()
        return lay.timings()["launches"]

    one, two = launches(8192), launches(8193)
    assert two == one + 1
    routed = torch.empty(T, 1, 2, pin_memory=pinned)
    lay.forward(hidden.numpy(), router_out=route.numpy(), out=out.numpy(), router_out_buf=routed.numpy())
    assert lay.timings()["launches"] == (one if most <= 8192 else two)
    got, o = torch.empty(T, H, device="cuda"), out.clone()
    lay.forward_dev(hidden.cuda(), T, got, d_router_in=route.cuda())
    lay.sync()
    assert torch.equal(got.cpu(), o)
    lay.close()


def test_copies_in_step(gpu_lib):
    """Eight passes of 4.2 MB of a layer whose copies are all there is: the copies in go first, and every copy out waits for one of them."""
    E, k, H, F, T = 8, 2, 512, 64, 16384
    rng = np.random.default_rng(3)
    lay = MoeLayer(E, k, H, F, activation=1, has_bias=False, max_tokens=T)
    for e in range(E):
        b = [np.full((F * H // 32, 17), 120, np.uint8) for _ in range(3)]
        for m in b:
            m[:, 1:] = rng.integers(0, 256, m[:, 1:].shape)
        lay.load_expert(e, *(m.reshape(-1) for m in b))
    hidden = torch.from_numpy(rng.standard_normal((T, H)).astype(np.float32)).pin_memory()
    route = torch.rand(T, k, 2)
    route[..., 0] = torch.rand(T, E).argsort(1)[:, :k].float()
    route = route.pin_memory()
    want = torch.empty(T, H, device="cuda")
    lay.forward_dev(hidden.cuda(), T, want, d_router_in=route.cuda())
    lay.sync()
    out, routed = torch.zeros(T, H).pin_memory(), torch.zeros(T, k, 2).pin_memory()
    for _ in range(2):
        out.zero_()
        lay.forward(hidden.numpy(), router_out=route.numpy(), out=out.numpy(), router_out_buf=routed.numpy())
        assert torch.equal(out, want.cpu()) and torch.equal(routed, route)
    bad = route.clone().pin_memory()
    bad[T - 1, 1, 0] = E
    with pytest.raises(CskError, match="out of range"):
        lay.forward(hidden.numpy(), router_out=bad.numpy(), out=out.numpy(), router_out_buf=routed.numpy())
    lay.forward(hidden.numpy(), router_out=route.numpy(), out=out.numpy(), router_out_buf=routed.numpy())
    assert torch.equal(out, want.cpu())
    lay.close()
