"""The certified fast router against the CPU restatement of the reference's sequential-chain router:
expert indices must be identical for every token, whichever of the two passes (fast logits accepted by
their error bounds, or the chain for the tokens they cannot separate) produced them."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from coalsack_b200 import MoeLayer, synth

pytestmark = pytest.mark.gpu


def _router_layer(E, k, H, Wg, rb, max_tokens, sigmoid=False):
    """A router-only layer with the certified pass switched on for every batch size (the default mode
    keeps it for batches of up to four tokens)."""
    lay = MoeLayer(E, k, H, 32, has_bias=False, sigmoid_gating=sigmoid, max_tokens=max_tokens)
    lay.set_router(Wg, rb)
    lay.set_router_mode(lay.ROUTER_CERTIFIED)
    return lay


def _cpu_router(port, h, Wg, rb, k, threads=16):
    parts = np.array_split(np.arange(h.shape[0]), threads)
    with ThreadPoolExecutor(threads) as ex:
        outs = list(ex.map(lambda idx: port.router(h[idx], Wg, rb, k) if len(idx) else np.zeros((0, k, 2), np.float32), parts))
    return np.concatenate(outs)


def test_certified_router_49152_tokens_of_the_120b_shape(gpu_lib, port):
    """49 152 tokens on the 128-expert router, routed in decode-sized batches of 1 to 128 tokens through
    the certified pass: indices bit-exact, routing weights within 2e-6, and only a few percent of
    the tokens needed the chain.  Then one 8192-token batch in each of the three modes."""
    import torch
    sh = synth.C2
    E, k, H = sh.num_experts, sh.top_k, sh.hidden
    Wg, rb = synth.router_weight(sh), synth.router_bias(sh)
    lay = _router_layer(E, k, H, Wg, rb, 8192)
    sizes = [128, 64, 32, 16, 8, 4, 2, 1, 100, 29]
    for rep in range(6):
        h = synth.hidden_states(sh, 8192, rep=rep)
        h_d = torch.from_numpy(h).cuda()
        ro_d = torch.empty((8192, k, 2), dtype=torch.float32, device="cuda")
        pos, i = 0, 0
        while pos < 8192:
            n = min(sizes[i % len(sizes)] if rep == 0 else 128, 8192 - pos)
            lay.route_dev(h_d[pos:pos + n], n, ro_d[pos:pos + n])
            pos += n
            i += 1
        torch.cuda.synchronize()
        lay.sync()
        got = ro_d.cpu().numpy()
        want = _cpu_router(port, h, Wg, rb, k)
        assert np.array_equal(got[..., 0], want[..., 0]), f"batch {rep}: expert indices differ"
        assert np.allclose(got[..., 1], want[..., 1], atol=2e-6)
    routed, chained = lay.router_stats()
    assert routed == 6 * 8192
    assert 0 < chained < 0.08 * routed, (routed, chained)
    print(f"certified router: {chained} of {routed} tokens recomputed by the chain ({100.0 * chained / routed:.2f} %)")
    for mode in (lay.ROUTER_CERTIFIED, lay.ROUTER_CHAIN, lay.ROUTER_AUTO):   # a prefill-sized batch in every mode
        lay.set_router_mode(mode)
        h = synth.hidden_states(sh, 8192, rep=7)
        got = lay.route(h)
        want = _cpu_router(port, h, Wg, rb, k)
        assert np.array_equal(got[..., 0], want[..., 0]) and np.allclose(got[..., 1], want[..., 1], atol=2e-6)
    lay.set_router_mode(lay.ROUTER_CHAIN)
    h = synth.hidden_states(sh, 64, rep=8)
    assert np.array_equal(lay.route(h)[..., 0], port.router(h, Wg, rb, k)[..., 0])
    lay.close()


@pytest.mark.parametrize("T", [1, 3, 8, 37, 64, 128, 700])
def test_certified_router_small_batches(gpu_lib, port, T):
    """Decode-sized and ragged batches, sigmoid gating included, on the C4 router (no bias, top-8)."""
    sh = synth.C4
    E, k, H = sh.num_experts, sh.top_k, sh.hidden
    Wg = synth.router_weight(sh)
    for sigmoid in (False, True):
        lay = _router_layer(E, k, H, Wg, None, 1024, sigmoid=sigmoid)
        for rep in range(3):
            h = synth.hidden_states(sh, T, rep=10 * T + rep)
            got = lay.route(h)
            want = port.router(h, Wg, None, k, sigmoid)
            assert np.array_equal(got[..., 0], want[..., 0]), (T, rep, sigmoid)
            assert np.allclose(got[..., 1], want[..., 1], atol=2e-6)
        lay.close()


def test_near_ties_take_the_chain_and_still_match(gpu_lib, port):
    """Gate rows in near-duplicate pairs (a tenth of the elements moved by parts in 2^-14, so the twins'
    logits differ by about 1e-5): for most tokens two of the best logits are closer than any error bound,
    the selection cannot be certified and the chain decides.  Tokens whose CPU logits tie exactly among the
    k+1 best are left out (the reference's order is unspecified there, moe_router_node.h:175-177)."""
    rng = np.random.default_rng(5)
    E, k, H, T = 64, 4, 1024, 128
    base = (rng.standard_normal((E // 2, H)) * 0.05).astype(np.float32)
    twin = base.copy()
    move = rng.random((E // 2, H)) < 0.1
    twin[move] *= np.float32(1.0 + 2.0 ** -14)
    Wg = np.ascontiguousarray(np.stack([base, twin], axis=1).reshape(E, H))
    rb = (rng.standard_normal(E) * 0.01).astype(np.float32)
    rb[1::2] = rb[0::2]
    h = rng.standard_normal((T, H)).astype(np.float32)
    lay = _router_layer(E, k, H, Wg, rb, T)
    got = lay.route(h)
    routed, chained = lay.router_stats()
    assert routed == T and chained > T // 2, (routed, chained)
    want, logits = port.router_logits(h, Wg, rb, k)
    top = -np.sort(-logits, axis=1)[:, :k + 1]
    clean = np.all(top[:, :-1] != top[:, 1:], axis=1)
    assert clean.sum() > T // 2
    assert np.array_equal(got[clean][..., 0], want[clean][..., 0])
    lay.close()


@pytest.mark.parametrize("E,k,H,T,kind", [
    (33, 4, 32, 2048, "normal"),     # one block of columns, half of it padding; two groups of 32, 95 of 128 rows padding
    (128, 8, 96, 1025, "normal"),    # a tile of one token; the last block half full
    (129, 2, 160, 1024, "heavy"),    # a second group of 128 experts with one row
    (160, 16, 2080, 1100, "heavy"),  # more parts of the hidden dimension than tiles of one wave
    (256, 1, 64, 4161, "tiny"),      # digits of blocks near the smallest scale
    (64, 6, 2880, 8192, "normal"),   # one part, every stage of the ring many times over
])
def test_certified_router_on_the_tensor_cores(gpu_lib, port, E, k, H, T, kind):
    """Large batches: the digits' logits and bounds, where tiles, groups and parts end.  Rows with an infinity or a NaN
    certify nothing, touch no other row, and go through the chain."""
    rng = np.random.default_rng(E + T)
    Wg = (rng.standard_normal((E, H)) * 0.05).astype(np.float32)
    h = rng.standard_normal((T, H)).astype(np.float32)
    if kind == "heavy":
        h, Wg = h ** 5, Wg * np.exp(rng.standard_normal((E, H))).astype(np.float32)
    if kind == "tiny":
        h[::3] *= np.float32(2.0 ** -100)
        h[1::3, : H // 2] = 0
    rb = None if kind == "heavy" else (rng.standard_normal(E) * 0.01).astype(np.float32)
    lay = _router_layer(E, k, H, Wg, rb, T)
    got = lay.route(h)
    want, logits = port.router_logits(h, Wg, rb, k)
    top = -np.sort(-logits, axis=1)[:, :k + 1]
    clean = np.all(top[:, :-1] != top[:, 1:], axis=1)   # the reference leaves the order of equal logits open
    assert clean.mean() > 0.6
    assert np.array_equal(got[clean][..., 0], want[clean][..., 0])
    # a softmax weight moves by at most the logits' errors: the chain's own (measured against 64 bits) and, of the
    # digits' sums, a few roundings; against 64 bits they are no further off than the chain
    exact = h.astype(np.float64) @ Wg.T.astype(np.float64) + (0 if rb is None else rb.astype(np.float64))
    chain_err = np.abs(logits - exact).max(1)
    tol = 2e-6 + 2 * chain_err
    assert np.all(np.abs(got[..., 1] - want[..., 1]).max(1)[clean] <= tol[clean])
    sel = np.take_along_axis(exact, want[..., 0].astype(np.int64), 1)
    w64 = np.exp(sel - sel.max(1, keepdims=True))
    w64 /= w64.sum(1, keepdims=True)
    off_got, off_want = (np.abs(r[clean][..., 1] - w64[clean]).mean() for r in (got, want))
    assert off_got <= 1.05 * off_want + 1e-9, (off_got, off_want)
    routed, chained = lay.router_stats()
    assert routed == T and chained < 0.8 * T
    bad = h.copy()
    bad[5, H - 1], bad[T - 1, 0] = np.inf, np.nan
    other = lay.route(bad)
    keep = clean.copy()
    keep[[5, T - 1]] = False
    assert np.array_equal(other[keep], got[keep])
    assert lay.router_stats()[1] - chained >= 2
    lay.close()


@pytest.mark.parametrize("T", [2, 2048])
def test_an_expert_left_out_with_a_large_bound_is_not_overlooked(gpu_lib, port, T):
    """One gate row's terms are rounded up next to a large entry that cancels at the end: its chain logit is twice the exact
    one, the highest of all, while its exact logit is only the fourth, behind three with small error bounds."""
    E, k, H = 40, 2, 64
    Wg = np.zeros((E, H), np.float32)
    Wg[0, 1], Wg[1, 1], Wg[2, 1] = 2.0, 1.9, 1.8
    Wg[5, 0], Wg[5, 62] = 2.0 ** 20, -(2.0 ** 20)
    Wg[5, np.r_[1:25:2, 33:57:2]] = 0.0626
    h = np.ones((T, H), np.float32)
    want, logits = port.router_logits(h, Wg, None, k)
    assert np.argmax(logits[0]) == 5 and abs(Wg[5].astype(np.float64).sum() - 24 * 0.0626) < 1e-6
    lay = _router_layer(E, k, H, Wg, None, T)
    assert np.array_equal(lay.route(h)[..., 0], want[..., 0])
    lay.close()


def test_tokens_whose_squares_underflow_are_not_certified_by_mistake(gpu_lib, port):
    """Token rows near 2^-78 whose logits cancel down to the size of the chain's own rounding errors: their norms' squares
    are below the smallest float, but the bounds must not be."""
    E, k, H, T = 64, 2, 64, 2048
    rng = np.random.default_rng(19)
    g = rng.standard_normal(H).astype(np.float32)
    Wg = rng.standard_normal((E, H)).astype(np.float32)
    Wg[:, -1] = (2.0 ** -17 * rng.standard_normal(E) - Wg[:, :-1].astype(np.float64) @ g[:-1].astype(np.float64)) / g[-1]
    h = (g * 2.0 ** -78 * rng.uniform(1, 2, (T, 1))).astype(np.float32)
    want, logits = port.router_logits(h, Wg, None, k)
    top = -np.sort(-logits, axis=1)[:, :k + 1]
    clean = np.all(top[:, :-1] != top[:, 1:], axis=1)
    exact = np.argsort(-(h.astype(np.float64) @ Wg.T.astype(np.float64)), axis=1)[:, :k]
    assert np.any(exact[clean] != want[clean][..., 0])  # the chain orders some tokens otherwise than exact arithmetic
    lay = _router_layer(E, k, H, Wg, None, T)
    assert np.array_equal(lay.route(h)[clean][..., 0], want[clean][..., 0])
    lay.close()


def test_lists_of_any_length_go_through_the_chain(gpu_lib, port):
    """Tokens that the certified pass cannot separate: a few, more than one round of the launch for short lists holds, and
    most of the batch (the other launch's), in turn on one handle; the experts are the reference's each time."""
    E, k, H, T = 64, 4, 256, 2048
    rng = np.random.default_rng(23)
    Wg = (rng.standard_normal((E, H)) * 0.05).astype(np.float32)
    Wg[E // 2:] = Wg[:E // 2]          # pairs of gate rows that differ in one column
    Wg[E // 2:, 40] += np.float32(1e-3)
    lay = _router_layer(E, k, H, Wg, None, T)
    before = 0
    for m in (30, 1500, 0, 500, T, 3):
        h = rng.standard_normal((T, H)).astype(np.float32)
        h[:, 40] = 4.0
        h[rng.permutation(T)[:m], 40] = 0.002     # their pairs of logits differ by 2e-6
        want, logits = port.router_logits(h, Wg, None, k)
        top = -np.sort(-logits, axis=1)[:, :k + 1]
        clean = np.all(top[:, :-1] != top[:, 1:], axis=1)
        assert clean.mean() > 0.9
        assert np.array_equal(lay.route(h)[clean][..., 0], want[clean][..., 0])
        chained = lay.router_stats()[1]
        assert m <= chained - before <= m + 0.1 * T, (m, chained - before)
        before = chained
    lay.close()


@pytest.mark.parametrize("E,T,certified", [(1024, 128, False), (1024, 256, True), (512, 511, False), (512, 512, True),
                                           (128, 1023, False), (128, 1024, True), (32, 4096, False)])
def test_which_batches_take_the_certified_pass_by_themselves(gpu_lib, port, E, T, certified):
    """The default mode's rule, on both sides of its line: the pass is taken where it is the faster of the two."""
    rng = np.random.default_rng(E + T)
    Wg = (rng.standard_normal((E, 64)) * 0.05).astype(np.float32)
    lay = _router_layer(E, 2, 64, Wg, None, T)
    lay.set_router_mode(lay.ROUTER_AUTO)
    h = rng.standard_normal((T, 64)).astype(np.float32)
    want, logits = port.router_logits(h, Wg, None, 2)
    top = -np.sort(-logits, axis=1)[:, :3]
    clean = np.all(top[:, :-1] != top[:, 1:], axis=1)
    assert np.array_equal(lay.route(h)[clean][..., 0], want[clean][..., 0])
    assert (lay.router_stats()[0] == T) == certified
    lay.close()


@pytest.mark.parametrize("E,k,H,T", [
    (5, 2, 2880, 3), (33, 4, 96, 1),         # an odd number of experts: their parts are copied one by one; one part
    (129, 8, 2880, 4), (1023, 16, 64, 2),    # a second and an eighth turn of a thread's experts
    (1024, 3, 4096, 4), (128, 16, 2880, 70), # the most parts x experts of a token; more tokens than one block of the logits
])
def test_certified_finish_edges(gpu_lib, port, E, k, H, T):
    """The certified pass of a few tokens where its loops over parts and experts end; a row of zeros goes through the chain."""
    rng = np.random.default_rng(E + H + T)
    Wg = (rng.standard_normal((E, H)) * 0.05).astype(np.float32)
    rb = (rng.standard_normal(E) * 0.01).astype(np.float32)
    h = rng.standard_normal((T, H)).astype(np.float32)
    h[T - 1] = 0
    for bias in (rb, None):
        lay = _router_layer(E, k, H, Wg, bias, T)
        got = lay.route(h)
        want = port.router(h, Wg, bias, k)
        rows = slice(None) if bias is not None else slice(0, T - 1)  # (without a bias the last row's logits are all equal: any order)
        assert np.array_equal(got[rows, :, 0], want[rows, :, 0])
        # A logit of either kind is within b = 2^-24 (sum of |partial sums| + sum of |terms|) of the exact one, so the difference of two logits
        # moves by no more than 4 b and a weight by that share of it (and by the rounding of exp and the division).
        terms = h[:, None].astype(np.float64) * Wg[got[..., 0].astype(int) % E]
        b = 2.0 ** -24 * (np.abs(np.cumsum(terms, -1)).sum(-1) + np.abs(terms).sum(-1)).max(-1, keepdims=True)
        assert (np.abs(got[..., 1] - want[..., 1])[rows] <= (want[..., 1] * (4 * b + 2e-6))[rows]).all()
        lay.close()
