"""fp16 weights on few token rows (the streaming kernel of the dense FFN and of fp16 experts) at the ends of its row groups,
k-tiles and warps, against the CPU restatement of the reference; and the first batch of the kernel after it."""
import numpy as np
import pytest
import torch

from coalsack_b200 import MoeLayer, dense_ffn_node, synth
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 8, 9, 16, 17, 32, 33, 64, 65])
@pytest.mark.parametrize("H,F,bias", [
    (32, 96, True),       # one k-tile of which half is padding: seven of eight warps idle
    (544, 160, False),    # nine k-tiles (the warps' second turn) and three
    (1088, 2080, True),   # seventeen and thirty-three: the third and fifth turn
    (96, 2368, True), (2400, 64, False),  # the most blocks that are resident at once with more than 32 rows, and too many
])
def test_dense(gpu_lib, port, H, F, bias, T):
    hidden, gw, uw, dw, bg, bu, bd = cases.dense_ffn_case(H=H, F=F, T=T, bias=True, seed=700 + T)
    biases = [bg, bu, bd] if bias else []
    node = dense_ffn_node()
    out = node.compute([hidden[None], gw, uw, dw] + biases)[0]
    mx, mr = cases.err_stats(out, port.dense_ffn(hidden, gw, uw, dw, *(biases or [None] * 3)))
    assert mx <= cases.MAX_ABS_OVER_RMS and mr <= cases.MEAN_REL, (mx, mr)
    assert np.array_equal(out, node.compute([hidden[None], gw, uw, dw] + biases)[0])
    node.close()


@pytest.mark.parametrize("E,k,T,wbf", [
    (5, 1, 3, False), (5, 2, 8, False), (5, 2, 9, True), (40, 2, 16, False), (40, 4, 16, True),  # the streaming kernel
    (5, 2, 17, False), (5, 2, 20, False), (40, 4, 64, True),                                  # the tensor-core kernel
])
def test_experts(gpu_lib, port, E, k, T, wbf):
    """Routed fp16 experts: more tiles than rows and fewer, experts without rows, a row that is not finite touches no other."""
    H, F = 288, 160
    rng = np.random.default_rng(E + T)
    hidden = rng.standard_normal((T, H)).astype(np.float32)
    experts = [cases.dense_ffn_case(H=H, F=F, T=1, bias=True, seed=900 + e)[1:] for e in range(E)]
    lay = MoeLayer(E, k, H, F, activation=synth.STANDARD_SWIGLU, has_bias=True, max_tokens=T, weights_f16=True, weight_before_ffn=wbf)
    lay.set_router((rng.standard_normal((E, H)) * 0.3).astype(np.float32), None)
    for e, (gw, uw, dw, bg, bu, bd) in enumerate(experts):
        lay.load_expert_f16(e, uw, gw, dw, bu, bg, bd)
    out, ro = lay.forward(hidden)
    want = np.zeros((T, H), np.float32)
    for j in range(k):
        w = ro[:, j, 1:]
        for e in set(ro[:, j, 0].astype(int)):
            on = ro[:, j, 0] == e
            want[on] += port.dense_ffn(w[on] * hidden[on], *experts[e]) if wbf else w[on] * port.dense_ffn(hidden[on], *experts[e])
    mx, mr = cases.err_stats(out, want)
    assert mx <= cases.MAX_ABS_OVER_RMS and mr <= cases.MEAN_REL, (mx, mr)
    bad = hidden.copy()
    bad[T // 2, 5] = np.inf
    got, _ = lay.forward(bad, router_out=ro)
    keep = np.arange(T) != T // 2
    assert np.array_equal(got[keep], out[keep]) and not np.isfinite(got[T // 2]).any()
    lay.close()


@pytest.mark.parametrize("E,count,k,T", [
    (5, 0, 2, 1), (5, 0, 2, 5), (5, 0, 2, 8), (5, 0, 2, 9), (5, 0, 4, 5), (5, 0, 4, 16),  # up to four turns of a tile's rows
    (16, 0, 16, 16),                                                                      # 256 rows: two tiles of one expert
    (4, 1, 2, 8), (4, 1, 4, 9), (4, 1, 4, 16), (4, 1, 4, 64),                             # a shard that holds one expert
])
@pytest.mark.parametrize("one", [True, False])
def test_routing_that_names_an_expert_twice(gpu_lib, port, E, count, k, T, one):
    """The caller's routing may fill several slots of a token with one expert (padding with expert 0 does): every such pair
    is a row of its own, so an expert has up to k rows per token.  After a batch of other values, whose rows must not show."""
    H, F = 288, 160
    held = count or E
    rng = np.random.default_rng(E + k + T)
    experts = [cases.dense_ffn_case(H=H, F=F, T=1, bias=True, seed=950 + e)[1:] for e in range(held)]
    lay = MoeLayer(E, k, H, F, activation=synth.STANDARD_SWIGLU, has_bias=True, max_tokens=80, weights_f16=True, expert_count=count)
    for e, (gw, uw, dw, bg, bu, bd) in enumerate(experts):
        lay.load_expert_f16(e, uw, gw, dw, bu, bg, bd)

    def routing(n):
        ro = rng.uniform(0.1, 1.0, (n, k, 2)).astype(np.float32)
        ro[..., 0] = 0 if one else rng.integers(0, held, (n, k))
        return ro

    def forward(hidden, ro):  # (on device buffers: never cut into passes)
        x, r, out = torch.from_numpy(hidden).cuda(), torch.from_numpy(ro).cuda(), torch.empty(hidden.shape, device="cuda")
        torch.cuda.synchronize()
        lay.forward_dev(x, len(hidden), out, d_router_in=r)
        lay.sync()
        return out.cpu().numpy()

    forward((100 * rng.standard_normal((80, H))).astype(np.float32), routing(80))
    hidden, ro = rng.standard_normal((T, H)).astype(np.float32), routing(T)
    out = forward(hidden, ro)
    dense = [port.dense_ffn(hidden, *w) for w in experts]
    want = np.zeros((T, H), np.float32)
    for j in range(k):
        want += ro[:, j, 1:] * np.stack([dense[int(e)][t] for t, e in enumerate(ro[:, j, 0])])
    mx, mr = cases.err_stats(out, want)
    assert mx <= cases.MAX_ABS_OVER_RMS and mr <= cases.MEAN_REL, (mx, mr)
    named = (ro[..., 0] == 0).any(axis=1)
    if named.any():
        alone = lay.expert_forward(0, hidden, ro)
        mx, mr = cases.err_stats(alone[named], dense[0][named])
        assert mx <= cases.MAX_ABS_OVER_RMS and mr <= cases.MEAN_REL, (mx, mr)
        assert np.all(alone[~named] == 0)
    lay.close()


@pytest.mark.parametrize("E,k,T,few", [(64, 8, 4, True), (64, 8, 15, False), (8, 2, 15, True)])
def test_many_hit_experts_go_to_the_tensor_core_kernel(gpu_lib, E, k, T, few):
    """The streaming kernel is the slower one once a small batch hits many experts.  The tensor-core kernel serves 17 tokens in
    any case, and a row's bits do not depend on its batch: so it has served the shorter batch if and only if the bits agree."""
    H, F = 256, 512
    rng = np.random.default_rng(E + T)
    lay = MoeLayer(E, k, H, F, activation=synth.STANDARD_SWIGLU, has_bias=False, max_tokens=17, weights_f16=True)
    for e in range(E):
        _, gw, uw, dw, *_ = cases.dense_ffn_case(H=H, F=F, T=1, bias=False, seed=e)
        lay.load_expert_f16(e, uw, gw, dw)
    hidden = rng.standard_normal((17, H)).astype(np.float32)
    ro = rng.uniform(0.1, 1.0, (17, k, 2)).astype(np.float32)
    ro[..., 0] = [rng.permutation(E)[:k] for _ in range(17)]
    out, _ = lay.forward(hidden, router_out=ro)
    short, _ = lay.forward(hidden[:T], router_out=ro[:T])
    assert np.allclose(short, out[:T], rtol=0, atol=2e-2 * out.std())
    assert np.array_equal(short, out[:T]) == (not few)
    lay.close()
