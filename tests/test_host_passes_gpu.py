"""How many passes the host entry point cuts a batch into, by the memory of its buffers and the work that a pass would have.

The last pass's launches tell its size: up to 8192 (token, expert) pairs are planned by one launch, more by two."""
import numpy as np
import pytest
import torch

from coalsack_b200 import MoeLayer

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
