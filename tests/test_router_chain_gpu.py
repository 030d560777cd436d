"""The order-faithful router kernel where its blocks, stages and clusters end, against the CPU restatement: the products and
sums are the reference's one after the other, so the selections are equal and the routing weights are, too, but for the
exponential's last bits."""
import numpy as np
import pytest

from coalsack_b200 import MoeLayer

pytestmark = pytest.mark.gpu


def _waves():
    """The last batch of each launch shape and the first of the next: of `tokens` a block, one wave of blocks (as many as the handle
    says are resident at once), and a token more."""
    for E in (32, 64, 128, 256):
        for tokens in (1, 2, 4, 8, 12, 16, 24, 32):
            yield E, 96, (tokens, 0)
            yield E, 96, (tokens, 1)


def _batch(E, H, T):
    """T, or the batch that a wave of `tokens` a block and `more` tokens make."""
    if not isinstance(T, tuple):
        return T
    lay = MoeLayer(E, 1, H, 32, has_bias=False, max_tokens=1)
    blocks = lay.debug_get(lay.DEBUG_ROUTER_WAVE)
    lay.close()
    return blocks // (-(-E // 32)) * T[0] + T[1]


@pytest.mark.parametrize("E,H,T", [
    *_waves(),
    (5, 32, 3), (33, 256, 7), (64, 288, 9),          # fewer columns than a stage, one stage, one more block of columns
    (256, 1056, 5), (257, 544, 5), (1024, 160, 40),  # the widest cluster, the first without one, the most experts
    (128, 2880, 8), (128, 2880, 333), (40, 4128, 150),
    (512, 96, 40), (513, 96, 40), (1000, 64, 700),   # the selection's forms for 512 and 1024 experts
])
@pytest.mark.parametrize("sigmoid", [False, True])
def test_chain_at_the_edges_of_its_launches(gpu_lib, port, E, H, T, sigmoid):
    T = _batch(E, H, T)
    rng = np.random.default_rng(E + H + T)
    k = min(4, E)
    h = rng.standard_normal((T, H)).astype(np.float32)
    Wg = (rng.standard_normal((E, H)) * 0.02).astype(np.float32)
    rb = (rng.standard_normal(E) * 0.01).astype(np.float32)
    lay = MoeLayer(E, k, H, 32, has_bias=False, sigmoid_gating=sigmoid, max_tokens=T)
    lay.set_router(Wg, rb)
    lay.set_router_mode(lay.ROUTER_CHAIN)
    got = lay.route(h)
    want = port.router(h, Wg, rb, k, sigmoid)
    assert np.array_equal(got[..., 0], want[..., 0])
    # expf: 2 ulp here, in its sum as much again, and the reciprocal's and the product's roundings: 2.4e-7 + 2.4e-7 + 1.2e-7 of a weight
    assert np.allclose(got[..., 1], want[..., 1], rtol=0, atol=6e-7)
    assert np.array_equal(lay.route(h), got)
    lay.close()


@pytest.mark.parametrize("E,H,T", [(2, 128, 1), (64, 1024, 4), (300, 160, 3), (1024, 96, 2)])
def test_a_handful_of_tokens_that_cannot_be_separated(gpu_lib, port, E, H, T):
    """Gate rows in pairs that differ in a few low bits: the bounds cannot tell them apart, and the tokens of a batch this small
    take the certified pass and then the chain.  (Tokens whose logits tie among the k + 1 best are left out.)"""
    rng = np.random.default_rng(E)
    k = min(4, E // 2)
    base = (rng.standard_normal((E // 2, H)) * 0.05).astype(np.float32)
    twin = base.copy()
    move = rng.random(base.shape) < 0.1
    twin[move] *= np.float32(1.0 + 2.0 ** -14)
    Wg = np.ascontiguousarray(np.stack([base, twin], axis=1).reshape(E, H))
    lay = MoeLayer(E, k, H, 32, has_bias=False, max_tokens=T)
    lay.set_router(Wg, None)
    seen = 0
    for rep in range(8):
        h = rng.standard_normal((T, H)).astype(np.float32)
        got = lay.route(h)
        want, logits = port.router_logits(h, Wg, None, k)
        top = -np.sort(-logits, axis=1)[:, :k + 1]
        clean = np.all(top[:, :-1] != top[:, 1:], axis=1)
        seen += int(clean.sum())
        assert np.array_equal(got[clean][..., 0], want[clean][..., 0])
    routed, chained = lay.router_stats()
    assert routed == 8 * T and chained >= T and seen >= T, (routed, chained, seen)
    lay.close()


@pytest.mark.parametrize("E,H,T", [(33, 256, 3), (64, 288, 64), (128, 2880, 1), (128, 256, 333), (128, 160, 1100), (256, 1056, 40), (256, 96, 2000),
                                   (256, 288, 480), (256, 288, 481), (256, 256, 481), (224, 288, 585)])  # (the last batches of one wave of clusters, the first of one without)
def test_the_same_without_clusters(gpu_lib, E, H, T):
    """Where no cluster can be resident the groups of experts of a token block meet in global memory: the same routing bit for bit, of the
    chain and of the certified pass with its list."""
    rng = np.random.default_rng(E + T)
    h = rng.standard_normal((T, H)).astype(np.float32)
    h[::3] = h[0]  # (rows that repeat ...
    h[T - 1] = 0.0     # ... and one that no bound can certify)
    Wg = (rng.standard_normal((E, H)) * 0.02).astype(np.float32)
    lay = MoeLayer(E, 4, H, 32, has_bias=False, max_tokens=T)
    lay.set_router(Wg, None)
    assert lay.debug_get(lay.DEBUG_ROUTER_CLUSTERS) == 1
    modes = (lay.ROUTER_CHAIN, lay.ROUTER_CERTIFIED, lay.ROUTER_AUTO)
    want = []
    for mode in modes:
        lay.set_router_mode(mode)
        want.append(lay.route(h))
    lay.debug_set(lay.DEBUG_NO_CLUSTERS, 1)
    assert lay.debug_get(lay.DEBUG_ROUTER_CLUSTERS) == 0
    for mode, w in zip(modes, want):
        lay.set_router_mode(mode)
        for _ in range(2):
            assert np.array_equal(lay.route(h), w), mode
    lay.close()


@pytest.mark.parametrize("E,step", [(512, 256), (1024, 256), (1024, 255), (1024, 511)])
def test_equal_logits_go_to_the_lower_expert(gpu_lib, port, E, step):
    """Experts that repeat every `step` gate rows (in one lane of the selection, or in others): the lowest of the best one's copies first."""
    rng = np.random.default_rng(E + step)
    H, T, k = 64, 50, 5
    base = (rng.standard_normal((step, H)) * 0.1).astype(np.float32)
    Wg = np.ascontiguousarray(base[np.arange(E) % step])
    lay = MoeLayer(E, k, H, 32, has_bias=False, max_tokens=T)
    lay.set_router(Wg, None)
    lay.set_router_mode(lay.ROUTER_CHAIN)
    h = rng.standard_normal((T, H)).astype(np.float32)
    got = lay.route(h)[..., 0].astype(int)
    logits = port.router_logits(h, base, None, 1)[1]
    order = np.argsort(-logits, axis=1, kind="stable")
    for t in range(T):
        want = [e for b in order[t, :k] for e in range(b, E, step)][:k]
        assert got[t].tolist() == want, t
    lay.close()


@pytest.mark.parametrize("E", [5, 32, 64])
@pytest.mark.parametrize("tokens", [1, 2, 4, 8, 12, 16, 24, 32])
@pytest.mark.parametrize("more", [0, 1])
def test_plain_weights_at_the_edges_of_their_launches(gpu_lib, port, E, tokens, more):
    """The entry point without a handle: the last batch of each launch shape (one wave of blocks of so many tokens) and the first of the
    next.  Blocks of 16 tokens have one form for one wave and another for more."""
    import torch
    lib = gpu_lib
    blocks = torch.cuda.get_device_properties(0).multi_processor_count
    T, H, k = blocks // (-(-E // 32)) * tokens + more, 160, 4
    rng = np.random.default_rng(E + T)
    h = rng.standard_normal((T, H)).astype(np.float32)
    Wg = (rng.standard_normal((E, H)) * 0.02).astype(np.float32)
    rb = (rng.standard_normal(E) * 0.01).astype(np.float32)
    h_d, w_d, b_d = (torch.from_numpy(x).cuda() for x in (h, Wg, rb))
    out = torch.full((T, k, 2), -1.0, device="cuda")
    torch.cuda.synchronize()
    assert lib.csk_moe_route_static(h_d.data_ptr(), T, H, w_d.data_ptr(), b_d.data_ptr(), E, k, 0, out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert lib.csk_moe_route_static_status() == 0
    got, want = out.cpu().numpy(), port.router(h, Wg, rb, k, False)
    assert np.array_equal(got[..., 0], want[..., 0])
    assert np.allclose(got[..., 1], want[..., 1], rtol=0, atol=6e-7)  # (as above)
