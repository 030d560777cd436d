"""The plan of a batch (rows per expert, row tiles, places) where its block, its pairs per thread and its two forms end: the
caller's routing, against the CPU restatement, and the counters."""
import numpy as np
import pytest
import torch

from coalsack_b200 import CskError, MoeLayer, PATH_STREAM, PATH_TILE, synth
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,k,T", [
    (1, 1, 1), (33, 4, 9),                       # fewer pairs than threads; experts in two warps
    (1024, 1, 3), (1024, 2, 700),                # a thread per expert, one and two pairs each
    (3, 2, 4096), (3, 2, 4097), (40, 8, 1025),   # the most pairs of one launch and the fewest of two
])
@pytest.mark.parametrize("path", [PATH_STREAM, PATH_TILE])
def test_plan_edges(gpu_lib, port, E, k, T, path):
    sh = synth.tiny(seed=E + T, E=E, k=k, H=32, F=32, T=T, has_bias=True)
    h, Wg, rb, ex = cases.layer_inputs(sh)
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    lay.set_path(path)
    rng = np.random.default_rng(T)
    ro = rng.uniform(0.1, 1.0, (T, k, 2)).astype(np.float32)
    ro[..., 0] = [rng.permutation(E)[:k] for _ in range(T)]
    h_d, out_d = torch.from_numpy(h).cuda(), torch.empty((T, 32), device="cuda")
    torch.cuda.synchronize()

    def forward(routing):  # (on device buffers: never cut into passes)
        r = torch.from_numpy(routing).cuda()
        torch.cuda.synchronize()
        lay.forward_dev(h_d, T, out_d, d_router_in=r)
        lay.sync()
        return out_d.cpu().numpy()

    out = forward(ro)
    want, _ = port.moe_layer(h, Wg, rb, ex, k, sh.act, router_out=ro)
    mx, mr = cases.err_stats(out, want)
    assert mx <= cases.MAX_ABS_OVER_RMS and mr <= cases.MEAN_REL, (mx, mr)
    rows, distinct, _ = lay.counters()
    assert np.array_equal(rows, np.bincount(ro[..., 0].astype(int).ravel(), minlength=E)) and distinct == (rows > 0).sum()
    bad = ro.copy()
    bad[T - 1, k - 1, 0] = E
    with pytest.raises(CskError, match="out of range"):
        forward(bad)
    assert np.array_equal(forward(ro), out)
    lay.close()


@pytest.mark.parametrize("E,k,T", [
    (4, 1, 31), (64, 8, 128), (64, 8, 129),      # one warp and a lane less; the most pairs with a thread each, and one token more
    (2, 1, 1000), (1024, 1, 1024),               # many tiles of an expert; as many experts as pairs
])
@pytest.mark.parametrize("path", [PATH_STREAM, PATH_TILE])
def test_plan_of_a_thread_per_pair(gpu_lib, port, E, k, T, path):
    """Rows that share an expert unevenly, some of it not loaded: outputs against the restatement, counters, and the error."""
    sh = synth.tiny(seed=E + T, E=E, k=k, H=64, F=32, T=T, has_bias=True)
    h, Wg, rb, ex = cases.layer_inputs(sh)
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex, range(E - 1))
    lay.set_path(path)
    rng = np.random.default_rng(T)
    ro = rng.uniform(0.1, 1.0, (T, k, 2)).astype(np.float32)
    p = 1.0 / (1.0 + np.arange(E - 1)) if E > 2 else np.ones(1)
    ro[..., 0] = [rng.choice(E - 1, k, replace=False, p=p / p.sum()) for _ in range(T)]
    h_d, out_d = torch.from_numpy(h).cuda(), torch.empty((T, 64), device="cuda")

    def forward(routing):
        r = torch.from_numpy(routing).cuda()
        torch.cuda.synchronize()
        lay.forward_dev(h_d, T, out_d, d_router_in=r)
        lay.sync()
        return out_d.cpu().numpy()

    out = forward(ro)
    want, _ = port.moe_layer(h, Wg, rb, ex, k, sh.act, router_out=ro)
    mx, mr = cases.err_stats(out, want)
    assert mx <= cases.MAX_ABS_OVER_RMS and mr <= cases.MEAN_REL, (mx, mr)
    rows, distinct, _ = lay.counters()
    assert np.array_equal(rows, np.bincount(ro[..., 0].astype(int).ravel(), minlength=E)) and distinct == (rows > 0).sum()
    absent = ro.copy()
    absent[0, 0, 0] = E - 1
    with pytest.raises(CskError, match="not loaded"):
        forward(absent)
    assert np.array_equal(forward(ro), out)
    lay.close()


@pytest.mark.parametrize("k", [4, 5, 8, 9, 16])  # slots asked for at once, and one more
def test_combine_adds_the_slots_in_order(gpu_lib, port, k):
    """Block calls (with a residual) and plain ones: the routed sum in router order, then the residual, bit for bit from one another."""
    sh = synth.tiny(seed=k, E=20, k=k, H=96, F=32, T=11, has_bias=True)
    h, Wg, rb, ex = cases.layer_inputs(sh, router_scale=30.0)
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    nw = np.ones(96, np.float32)
    lay.set_ffn_norm(nw, 1e-5)
    n = port.rmsnorm(h, nw, 1e-5)
    out, ro = lay.forward(n)
    want, _ = port.moe_layer(n, Wg, rb, ex, k, sh.act, router_out=ro)
    mx, mr = cases.err_stats(out, want)
    assert mx <= cases.MAX_ABS_OVER_RMS and mr <= cases.MEAN_REL, (mx, mr)
    block, ro2 = lay.block_forward(h)
    assert np.array_equal(ro, ro2) and np.array_equal((h + out).astype(np.float32), block)
    lay.close()


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("T", [7, 700, 1500])  # fewer tokens than four an SM, than five, and more than six: two forms of the combine
def test_merge_adds_the_slots_one_after_the_other(gpu_lib, k, T):
    """Rows of very different size, so that another order gives other bits: equal to products and sums in fp32, slot by slot."""
    E, H = k + 3, 96
    rng = np.random.default_rng(100 * k + T)
    y = (rng.standard_normal((E, T, H)) * 10.0 ** rng.uniform(-3, 3, (E, T, 1))).astype(np.float32)
    ro = rng.uniform(0.1, 1.0, (T, k, 2)).astype(np.float32)
    ro[..., 0] = [rng.permutation(E)[:k] for _ in range(T)]
    absent = int(ro[0, k - 1, 0]) if k > 1 else E - 1  # an expert without output adds nothing
    lay = MoeLayer(E, k, H, 32, has_bias=False, max_tokens=T)
    got = lay.merge(ro, [None if e == absent else y[e] for e in range(E)])

    def in_order(slots):
        acc = np.zeros((T, H), np.float32)
        for j in slots:
            e = ro[:, j, 0].astype(int)
            term = ro[:, j, 1:] * y[e, np.arange(T)]
            acc = np.where((e != absent)[:, None], acc + term, acc)
        return acc

    assert np.array_equal(got, in_order(range(k)))
    assert k < 4 or not np.array_equal(got, in_order(reversed(range(k))))
    lay.close()


@pytest.mark.parametrize("k", [1, 4, 5, 8, 16])
@pytest.mark.parametrize("T", [11, 700, 1500])
def test_shared_and_residual_rows_come_last(gpu_lib, port, k, T):
    """A block call with a shared expert: x + (routed sum + shared expert's row), bit for bit from the parts."""
    H = 96
    sh = synth.tiny(seed=40 + k, E=20, k=k, H=H, F=32, T=T, has_bias=True)
    h, Wg, rb, ex = cases.layer_inputs(sh, router_scale=30.0)
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    nw = (1.0 + 0.1 * np.random.default_rng(k).standard_normal(H)).astype(np.float32)
    lay.set_ffn_norm(nw, 1e-5)
    _, gw, uw, dw, bg, bu, bd = cases.dense_ffn_case(H=H, F=64, T=1, bias=True, seed=k)
    shared = MoeLayer(1, 1, H, 64, activation=synth.STANDARD_SWIGLU, has_bias=True, max_tokens=T, weights_f16=True)
    shared.load_expert_f16(0, uw, gw, dw, bu, bg, bd)
    n = port.rmsnorm(h, nw, 1e-5)
    x_d, n_d = torch.from_numpy(h).cuda(), torch.from_numpy(n).cuda()
    block, moe, dense = (torch.empty((T, H), device="cuda") for _ in range(3))
    ro, ro2 = (torch.empty((T, k, 2), device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    for with_shared in (shared, None):
        lay.block_forward_dev(x_d, T, ro, block, shared=with_shared)
        lay.sync()
        lay.forward_dev(n_d, T, moe, d_router_out=ro2)
        lay.sync()
        shared.dense_forward_dev(n_d, T, dense)
        shared.sync()
        assert torch.equal(ro, ro2)
        want = moe + dense if with_shared else moe
        assert torch.equal(block, x_d + want)
    shared.close()
    lay.close()


@pytest.mark.parametrize("T", [1, 9, 200, 256, 257])  # up to 1024 pairs a thread each, then one block's histogram
@pytest.mark.parametrize("path", [PATH_STREAM, PATH_TILE])
def test_plan_of_a_shard(gpu_lib, T, path):
    """A handle that holds experts 8 to 15 of 24: rows of the others, on both sides, are counted and take no tiles.  Tokens whose experts are
    all here have the whole layer's results bit for bit."""
    E, k, H, first, held = 24, 4, 64, 8, 8
    sh = synth.tiny(seed=T, E=E, k=k, H=H, F=32, T=T, has_bias=True)
    h, Wg, rb, ex = cases.layer_inputs(sh)
    rng = np.random.default_rng(T)
    ro = rng.uniform(0.1, 1.0, (T, k, 2)).astype(np.float32)
    here = np.arange(T) % 2 == 0
    ro[..., 0] = [first + rng.permutation(held)[:k] if x else rng.permutation(E)[:k] for x in here]
    h_d, r_d = torch.from_numpy(h).cuda(), torch.from_numpy(ro).cuda()
    outs, rows = [], []
    for shard in (False, True):
        lay = MoeLayer.from_shape(sh, expert_begin=first, expert_count=held) if shard else MoeLayer.from_shape(sh)
        lay.set_router(Wg, rb)
        if shard:
            lay.load_experts({n: w[first:first + held] for n, w in ex.items()}, range(first, first + held))
        else:
            lay.load_experts(ex)
        lay.set_path(path)
        out = torch.empty((T, H), device="cuda")
        torch.cuda.synchronize()
        lay.forward_dev(h_d, T, out, d_router_in=r_d)
        lay.sync()
        outs.append(out.cpu().numpy())
        rows.append(lay.counters()[0])
        lay.close()
    assert np.array_equal(outs[1][here], outs[0][here])
    want = np.bincount(ro[..., 0].astype(int).ravel(), minlength=E)
    assert np.array_equal(rows[0], want) and np.array_equal(rows[1], want)


def test_more_rows_than_the_images_hold(gpu_lib):
    """An expert node's routing may name its expert in every slot, which makes more rows than a shard of one expert has images
    for: an error, and the handle goes on."""
    E, k, H, e = 8, 8, 64, 3
    sh = synth.tiny(seed=5, E=E, k=k, H=H, F=64, T=64, has_bias=True)
    h, _, _, ex = cases.layer_inputs(sh)
    lay = MoeLayer.from_shape(sh, expert_begin=e, expert_count=1)
    lay.load_experts(ex, [e])

    def routing(T, slots):
        ro = np.ones((T, k, 2), np.float32)
        ro[..., 0] = np.where(np.arange(k) < slots, e, 0)
        return ro

    once = lay.expert_forward(e, h[:10], routing(10, 1))  # 10 rows
    assert np.array_equal(lay.expert_forward(e, h[:2], routing(2, k)), once[:2])  # 16 rows
    with pytest.raises(CskError):
        lay.expert_forward(e, h[:10], routing(10, k))  # 80 rows
    assert np.array_equal(lay.expert_forward(e, h[:10], routing(10, 1)), once)
    lay.close()
