"""Calls enqueued one behind the other on one stream, each with its own tokens and no wait between them: every kernel may be resident
before the one in front has ended, and reads ahead of its wait what is older than that.  The results are bit for bit those of the
same calls with the device waited for in between."""
import numpy as np
import pytest
import torch

from coalsack_b200 import MoeLayer, synth
from tests import cases

pytestmark = pytest.mark.gpu

CALLS = 6


def _mxfp4(E, k, H, F, T):
    sh = synth.tiny(seed=E + T, E=E, k=k, H=H, F=F, T=T, has_bias=True)
    _, Wg, rb, ex = cases.layer_inputs(sh)
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    return lay


def _f16(E, k, H, F, T):
    lay = MoeLayer(E, k, H, F, activation=1, has_bias=False, max_tokens=T, weights_f16=True)
    rng = np.random.default_rng(E + T)
    for e in range(E):
        lay.load_expert_f16(e, *((rng.standard_normal(s) * s[1] ** -0.5).astype(np.float16) for s in ((F, H), (F, H), (H, F))))
    lay.set_router((rng.standard_normal((E, H)) * 0.1).astype(np.float32), None)
    return lay


@pytest.mark.parametrize("make,E,k,T", [
    (_mxfp4, 8, 2, 700),     # chain router in one group, plan in one block, CTA pairs
    (_mxfp4, 64, 2, 2100),   # certified router on tensor cores
    (_mxfp4, 64, 4, 2100),   # more than 8192 pairs: a plan of two launches
    (_mxfp4, 128, 4, 600),   # clusters of four in the router; block-scaled kernel
    (_f16, 4, 2, 700),       # fp16 weights on CTA pairs
    (_f16, 1, 1, 600),
])
@pytest.mark.parametrize("entry", ["layer", "given", "block", "dense", "sent"])
def test_calls_behind_one_another(gpu_lib, make, E, k, T, entry):
    if entry == "dense" and E > 1:
        pytest.skip("the dense entry takes layers of one expert")
    H, F = 256, 160
    lay = make(E, k, H, F, T)
    lay.set_ffn_norm(np.linspace(0.5, 1.5, H, dtype=np.float32))
    g = torch.Generator(device="cuda")
    g.manual_seed(T)
    xs = [torch.randn(T, H, device="cuda", generator=g) for _ in range(CALLS)]
    routes = [torch.rand(T, k, 2, device="cuda", generator=g) for _ in range(CALLS)]
    for r in routes:
        r[..., 0] = torch.rand(T, E, device="cuda", generator=g).argsort(1)[:, :k].float()
    ro = torch.empty(T, k, 2, device="cuda")
    send, back = torch.zeros(T * k, lay.ep_row_pitch(), dtype=torch.float16, device="cuda"), torch.empty(T * k, H, device="cuda")
    counts = torch.empty(E, dtype=torch.int32, device="cuda")
    tokens = [T, T - 1, T, T // 2 + 200, T, T - 33]

    def call(i, x, out):
        if entry == "layer":
            lay.forward_dev(x, tokens[i], out, d_router_out=ro)
        elif entry == "given":
            lay.forward_dev(x, tokens[i], out, d_router_in=routes[i])
        elif entry == "block":
            lay.block_forward_dev(x, tokens[i], ro, out)
        elif entry == "dense":
            lay.dense_forward_dev(x, tokens[i], out)
        else:  # the expert-parallel stages of one rank
            lay.ep_dispatch_dev(x, tokens[i], send, counts, d_router_in=routes[i] if i % 2 else None)
            lay.ep_experts_dev(send, counts, 1, tokens[i] * k, back)
            lay.ep_combine_dev(back, tokens[i], out)

    def run(wait, chained):
        outs = [torch.zeros(T, H, device="cuda") for _ in range(CALLS)]
        torch.cuda.synchronize()
        for i in range(CALLS):
            # chained: a call's rows are the next one's tokens, written by the last kernel in front of its first
            call(i, outs[i - 1] if chained and i else xs[i], outs[i])
            if wait:
                lay.sync()
        lay.sync()
        return [o.cpu() for o in outs]

    for chained in (False, True):
        want = run(True, chained)
        for _ in range(3):
            for i, (a, b) in enumerate(zip(run(False, chained), want)):
                assert torch.equal(a, b), (chained, i, (a != b).any(1).sum().item())
    lay.close()


@pytest.mark.parametrize("E,T", [(8, 3), (128, 4), (128, 64), (64, 2100), (300, 40)])
def test_routings_behind_one_another(gpu_lib, E, T):
    lay = MoeLayer(E, 4, 256, 32, has_bias=False, max_tokens=T)
    rng = np.random.default_rng(E + T)
    lay.set_router((rng.standard_normal((E, 256)) * 0.1).astype(np.float32), None)
    xs = [torch.from_numpy(rng.standard_normal((T, 256)).astype(np.float32)).cuda() for _ in range(CALLS)]
    for x in xs:
        x[::2] = x[0]  # (and rows that repeat)
    want, got = ([torch.zeros(T, 4, 2, device="cuda") for _ in range(CALLS)] for _ in range(2))
    torch.cuda.synchronize()
    for x, r in zip(xs, want):
        lay.route_dev(x, T, r)
        torch.cuda.synchronize()
    for _ in range(3):
        for x, r in zip(xs, got):
            lay.route_dev(x, T, r)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    lay.close()
