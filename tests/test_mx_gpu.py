"""The block-scaled expert kernel (weights as MXFP4 operands, token rows as five E2M1 digits) where its tiles, records and
padding end, against the CPU restatement of the reference."""
import numpy as np
import pytest

from coalsack_b200 import MoeLayer, PATH_STREAM, PATH_TILE, synth
from tests import cases

pytestmark = pytest.mark.gpu

# A block's digits leave at most 2^-14.2 of its largest value (0.2 of what an fp16 operand leaves, in norm); two
# contractions and fp32 sums in another order stay well under 1e-3 of the output's RMS.
MX_MAX, MX_MEAN = 2e-3, 3e-4


@pytest.mark.parametrize("E,k,H,F,T,bias,act,wbf", [
    (2, 1, 32, 32, 1, False, 0, False),      # one block: half of the K = 64 step is padding, 32 of 128 rows exist
    (2, 2, 96, 160, 3, True, 1, False),      # odd block counts either way; 15 of 16 columns
    (1, 1, 128, 128, 48, True, 0, False),    # two even tiles, one whole record
    (1, 1, 128, 128, 40, False, 1, False),   # one full tile (200 and 240 columns)
    (1, 1, 160, 384, 49, True, 0, True),     # two even tiles; second half of a plain unit absent; routing weight first
    (1, 1, 256, 288, 18, False, 0, False),   # the last height at which two units' accumulators fit in the down projection ...
    (1, 1, 256, 288, 19, False, 1, False),   # ... and the first at which they do not
    (1, 1, 256, 288, 22, False, 0, False),   # the same of gate/up ...
    (1, 1, 256, 288, 23, False, 1, False),   # ... and its first without
    (2, 1, 64, 4224, 60, False, 1, False),   # more than 32 records of activated rows: two mask words
    (3, 2, 288, 352, 145, True, 0, False),   # several tiles per expert, uneven loads
    (32, 2, 1536, 1536, 320, True, 0, False),  # several units per CTA, of tiles that do and that do not fit beside each other
    (4, 2, 2080, 1056, 65, True, 1, False),  # more records than ring stages
    (2, 1, 4128, 32, 5, False, 0, False),    # more than 128 blocks per row
])
def test_edges(gpu_lib, port, E, k, H, F, T, bias, act, wbf):
    sh = synth.tiny(seed=300 + T, E=E, k=k, H=H, F=F, T=T, has_bias=bias, act=act)
    h, Wg, rb, ex = cases.layer_inputs(sh, router_scale=30.0)
    lay = MoeLayer.from_shape(sh, weight_before_ffn=wbf)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    lay.set_path(PATH_STREAM)
    out, ro = lay.forward(h)
    want, want_ro = port.moe_layer(h, Wg, rb, ex, k, act, weight_before_ffn=wbf)
    assert np.array_equal(ro[..., 0], want_ro[..., 0])
    mx, mr = cases.err_stats(out, want)
    assert mx <= MX_MAX and mr <= MX_MEAN, (mx, mr)
    again, _ = lay.forward(h)
    assert np.array_equal(out, again)
    # a row that is not finite touches no other row, and nothing is left of it afterwards
    bad = h.copy()
    bad[T // 2, H - 1] = np.inf
    got, _ = lay.forward(bad, router_out=ro)
    keep = np.arange(T) != T // 2
    assert np.array_equal(got[keep], out[keep])
    after, _ = lay.forward(h)
    assert np.array_equal(after, out)
    lay.close()


@pytest.mark.parametrize("H", [384, 2080])  # the down projection's last unit has 128 rows, or 32, and no second half
@pytest.mark.parametrize("rows", [21, 22, 25, 26])  # the last with one atom of row scales and the first with two: down, gate/up
def test_units_without_a_second_half_beside_ordinary_ones(gpu_lib, port, H, rows):
    """Every expert has the same rows, so all tiles are alike; more units than CTAs, so that one CTA takes units of either kind."""
    E, F = 80 if H == 384 else 40, 192
    sh = synth.tiny(seed=rows, E=E, k=1, H=H, F=F, T=E * rows, has_bias=True)
    h, Wg, rb, ex = cases.layer_inputs(sh)
    ro = np.ones((E * rows, 1, 2), np.float32)
    ro[:, 0, 0] = np.random.default_rng(rows).permutation(np.repeat(np.arange(E), rows))
    ro[:, 0, 1] = 0.7
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    lay.set_path(PATH_STREAM)
    out, _ = lay.forward(h, router_out=ro)
    want, _ = port.moe_layer(h, Wg, rb, ex, 1, sh.act, router_out=ro, nthreads=16)
    mx, mr = cases.err_stats(out, want)
    assert mx <= MX_MAX and mr <= MX_MEAN, (mx, mr)
    lay.close()


@pytest.mark.parametrize("H,T", [(1056, 7), (2080, 7), (2880, 7),  # two and three CTAs a token, tails inside a warp
                                 (1056, 2800)])                    # rows that are claimed, one CTA a token
def test_routing_weight_before_the_expert(gpu_lib, H, T):
    """Rows encoded per pair, wide blocks among them: bit for bit the sum, slot by slot, of the results for rows that were weighted
    beforehand; of one expert alone, which leaves other slots' rows unplaced, its own."""
    E, k, F = 6, 3, 64
    sh = synth.tiny(seed=T + H, E=E, k=k, H=H, F=F, T=T, has_bias=True)
    h, _, _, ex = cases.layer_inputs(sh)
    h[T // 2, [5, H // 2, H - 3]] = 1000.0  # wide blocks, one of them the last
    rng = np.random.default_rng(H)
    ro = rng.uniform(0.1, 1.0, (T, k, 2)).astype(np.float32)
    ro[..., 0] = [rng.permutation(E)[:k] for _ in range(T)]

    def layer(k, before):
        lay = MoeLayer(E, k, H, F, activation=sh.act, has_bias=True, max_tokens=T, weight_before_ffn=before)
        lay.load_experts(ex)
        lay.set_path(PATH_STREAM)
        return lay

    first, plain = layer(k, True), layer(1, False)
    out, _ = first.forward(h, router_out=ro)
    want, parts = np.zeros_like(out), []
    for j in range(k):
        one = np.ones((T, 1, 2), np.float32)
        one[:, 0, 0] = ro[:, j, 0]
        parts.append(plain.forward(h * ro[:, j, 1:], router_out=one)[0])
        want = want + parts[-1]
    assert np.array_equal(out, want)
    if T < 100:
        e = int(ro[T // 2, 1, 0])
        alone = first.expert_forward(e, h, ro)
        for t, j in np.argwhere(ro[..., 0] == e):
            assert np.array_equal(alone[t], parts[j][t]), t
    first.close()
    plain.close()


def test_a_captured_step_outlives_larger_images(gpu_lib, port):
    """The digit images grow when the streaming kernel is chosen for any batch; a step that a caller captured before
    that still replays to the same result, on the images it was captured with."""
    import torch
    sh = synth.tiny(seed=351, E=2, k=1, H=256, F=192, T=160, has_bias=True)  # more rows than the first images hold
    h, Wg, rb, ex = cases.layer_inputs(sh, router_scale=30.0)
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    n = 24
    h_d, out = torch.from_numpy(h).cuda(), torch.empty((160, 256), device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    lay.forward_dev(h_d, n, torch.empty_like(out), stream=s.cuda_stream)  # (a call's own graph cannot be replayed in a capture)
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        lay.forward_dev(h_d, n, out, stream=s.cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    first = out[:n].cpu().numpy()
    want, _ = port.moe_layer(h, Wg, rb, ex, 1, sh.act)
    mx, mr = cases.err_stats(first, want[:n])
    assert mx <= MX_MAX and mr <= MX_MEAN, (mx, mr)
    lay.set_path(PATH_STREAM)
    whole, _ = lay.forward(h)
    mx, mr = cases.err_stats(whole, want)
    assert mx <= MX_MAX and mr <= MX_MEAN, (mx, mr)
    out.zero_()
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out[:n].cpu().numpy(), first)
    lay.close()


def test_received_rows_without_images_take_the_tensor_core_kernel(gpu_lib, port):
    """A layer that holds every expert has images for its own small batches only; the expert-parallel receive side may
    get more rows than those, allocates nothing, and takes the other kernel."""
    import torch
    from tests.test_ep_gpu import run_emulated_p2p
    sh = synth.tiny(seed=353, E=2, k=1, H=256, F=192, T=1, has_bias=True)
    _, Wg, rb, ex = cases.layer_inputs(sh, router_scale=30.0)
    for out, ro, hs in run_emulated_p2p(torch, sh, 1, (150,), Wg, rb, ex, 0):
        want, want_ro = port.moe_layer(hs, Wg, rb, ex, 1, sh.act)
        assert np.array_equal(ro[..., 0], want_ro[..., 0])
        mx, mr = cases.err_stats(out, want)
        assert mx <= cases.MAX_ABS_OVER_RMS and mr <= cases.MEAN_REL, (mx, mr)


# ---- operand precision where a few values of a block are far above the others -----------------------------------------
E2M1 = np.array([0, .5, 1, 1.5, 2, 3, 4, 6, 0, -.5, -1, -1.5, -2, -3, -4, -6])


def _values(blocks, rows, cols):
    """The numbers of an MXFP4 matrix in 64 bits."""
    b = np.asarray(blocks).reshape(rows, cols // 32, 17)
    codes = np.concatenate([b[:, :, 1:] & 15, b[:, :, 1:] >> 4], axis=2)
    return (E2M1[codes] * 2.0 ** (b[:, :, :1].astype(np.float64) - 127)).reshape(rows, cols)


def _zero_columns(blocks, rows, cols, which):
    b = np.asarray(blocks).reshape(rows, cols // 32, 17).copy()
    for c in which:
        j = c % 32
        b[:, c // 32, 1 + j % 16] &= 0xF0 if j < 16 else 0x0F
    return b.reshape(-1)


def _mlp64(h, ex, H, F, act):
    up, gate, down = (_values(ex[n][0], *s) for n, s in (("w_up", (F, H)), ("w_gate", (F, H)), ("w_down", (H, F))))
    u, g = h.astype(np.float64) @ up.T + ex["b_up"][0], h.astype(np.float64) @ gate.T + ex["b_gate"][0]
    if act == 0:
        g, u = np.minimum(g, 7), np.clip(u, -7, 7)
        a = g / (1 + np.exp(np.minimum(-1.702 * g, 700))) * (u + 1)
    else:
        a = g / (1 + np.exp(-g)) * u
    return a @ down.T + ex["b_down"][0]


@pytest.mark.parametrize("times", [1, 30, 100, 1000, 10000])
@pytest.mark.parametrize("where", ["dense", "unread", "activated"])
def test_outliers_lose_no_precision(gpu_lib, where, times):
    """Token rows with a few channels `times` above the others -- whose weights are ordinary, or zero, so that the others
    decide -- and a few activated features above the others that the down projection does not read: the result is no
    further from the 64-bit value than that of the kernel with fp16 operands (2e-6: fp32 sums of 1600 products)."""
    H, F, T, act = 1600, 480, 50, 1 if where == "activated" else 0
    sh = synth.tiny(seed=371, E=1, k=1, H=H, F=F, T=T, has_bias=True, act=act)
    h, Wg, rb, ex = cases.layer_inputs(sh)
    rng = np.random.default_rng(times)
    ex["w_gate"], ex["w_up"] = ([_scaled(w[0], -4)] for w in (ex["w_gate"], ex["w_up"]))
    if where == "activated":  # a handful of features at about `times` the others' values, their down columns zero
        big = rng.choice(F, 5, replace=False)
        ex["b_gate"][0][big], ex["b_up"][0][big] = 6.0, 0.5 * times
        ex["w_down"][0] = _zero_columns(ex["w_down"][0], H, F, big)
    else:
        big = rng.choice(H, 9, replace=False)
        h[:, big] = np.float32(times) * (1 + 0.1 * rng.standard_normal((T, 9))).astype(np.float32)
        if times > 1:
            h[:, big[0]] = times  # (an fp16 operand holds this one exactly)
        for n in ("w_gate", "w_up"):
            if where == "unread":
                ex[n][0] = _zero_columns(ex[n][0], F, H, big)
    want = _mlp64(h, ex, H, F, act)
    err = {}
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    route = np.zeros((T, 1, 2), np.float32)
    route[..., 1] = 1
    for name, path in (("fp16", PATH_TILE), ("digits", PATH_STREAM)):
        lay.set_path(path)
        out, _ = lay.forward(h, router_out=route)
        err[name] = np.linalg.norm(out - want) / np.linalg.norm(want)
        again, _ = lay.forward(h, router_out=route)
        assert np.array_equal(out, again)
    print(f"{where} x{times}: relative error fp16 operands {err['fp16']:.2e}, digits {err['digits']:.2e}")
    assert err["digits"] <= err["fp16"] + 2e-6, err
    # rows without outliers beside rows with them: the same bits as without
    if where != "activated":
        plain = synth.hidden_states(sh)
        alone, _ = lay.forward(plain, router_out=route)
        mixed = plain.copy()
        mixed[::3] = h[::3]
        both, _ = lay.forward(mixed, router_out=route)
        keep = np.arange(T) % 3 != 0
        assert np.array_equal(both[keep], alone[keep])
    lay.close()


@pytest.mark.parametrize("where", ["rows", "activated"])
def test_wide_blocks_past_the_first_word_of_marks(gpu_lib, where):
    """33 records: only the last one, marked in the second word, holds wide blocks (channels at 10^4 times the others that nothing reads).
    Without its second run those blocks' other values would be off by 10 %."""
    H, F, T = (4224, 64, 9) if where == "rows" else (64, 4224, 9)
    act = 0 if where == "rows" else 1
    sh = synth.tiny(seed=377, E=1, k=1, H=H, F=F, T=T, has_bias=True, act=act)
    h, Wg, rb, ex = cases.layer_inputs(sh)
    ex["w_gate"], ex["w_up"] = ([_scaled(w[0], -4)] for w in (ex["w_gate"], ex["w_up"]))
    big = np.array([4100, 4133, 4170, 4200])
    if where == "rows":
        h[:, big] = 1e4
        for n in ("w_gate", "w_up"):
            ex[n][0] = _zero_columns(ex[n][0], F, H, big)
    else:
        ex["b_gate"][0][big], ex["b_up"][0][big] = 6.0, 5e3
        ex["w_down"][0] = _zero_columns(ex["w_down"][0], H, F, big)
    want = _mlp64(h, ex, H, F, act)
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    route = np.zeros((T, 1, 2), np.float32)
    route[..., 1] = 1
    err = {}
    for name, path in (("fp16", PATH_TILE), ("digits", PATH_STREAM)):
        lay.set_path(path)
        out, _ = lay.forward(h, router_out=route)
        err[name] = np.linalg.norm(out - want) / np.linalg.norm(want)
    assert err["digits"] <= err["fp16"] + 2e-6, err  # (as above)
    lay.close()


def _scaled(blocks, by):
    """The matrix times 2^by."""
    b = np.asarray(blocks).reshape(-1, 17).copy()
    b[:, 0] = b[:, 0].astype(int) + by
    return b.reshape(-1)


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("path", [PATH_STREAM, PATH_TILE])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_a_row_that_is_not_finite_does_not_come_out_finite(gpu_lib, port, act, path, bad):
    """With the routing given by the caller nothing before the experts looks at the row: where the restatement's result is
    not finite, neither is the kernels' (the clamped activation keeps a NaN of the up projection), and no other row changes."""
    sh = synth.tiny(seed=361, E=2, k=1, H=160, F=96, T=9, has_bias=True, act=act)
    h, Wg, rb, ex = cases.layer_inputs(sh)
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    lay.set_path(path)
    route = np.ones((sh.tokens, 1, 2), np.float32)
    route[:, 0, 0] = np.arange(sh.tokens) % 2
    good, _ = lay.forward(h, router_out=route)
    h[4, 77] = bad
    out, _ = lay.forward(h, router_out=route)
    want, _ = port.moe_layer(h, Wg, rb, ex, 1, act, router_out=route)
    assert not np.isfinite(want[4]).any()
    assert not np.isfinite(out[4]).any()
    keep = np.arange(sh.tokens) != 4
    assert np.array_equal(out[keep], good[keep])
    lay.close()


@pytest.mark.parametrize("which", ["experts", "router"])
def test_waits_run_out_and_the_handle_recovers(gpu_lib, port, which):
    """The block-scaled kernel and the tensor-core router with a copy role that issues nothing, under a wait budget of 0.1 ms:
    every role gives up, the call reports it, and the same handle then computes the layer as before."""
    from coalsack_b200 import CskError
    T = 70 if which == "experts" else 2048
    sh = synth.tiny(seed=363, E=64, k=2, H=160, F=96, T=T, has_bias=True)
    h, Wg, rb, ex = cases.layer_inputs(sh, router_scale=30.0)
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    lay.set_path(PATH_STREAM)
    good, ro = lay.forward(h)
    assert which == "experts" or lay.router_stats()[0] == T  # the certified pass ran
    try:
        lay.debug_set(lay.DEBUG_WAIT_BUDGET, 200_000)
        lay.debug_set(lay.DEBUG_STALL_ROUTER if which == "router" else lay.DEBUG_STALL_TILE_PRODUCER, 1)
        with pytest.raises(CskError) as err:
            lay.forward(h)
        assert err.value.code == -3 and "wait ran out" in str(err.value)
    finally:
        lay.debug_set(lay.DEBUG_WAIT_BUDGET, 2_000_000_000)
    again, ro2 = lay.forward(h)
    assert np.array_equal(ro, ro2) and np.array_equal(good, again)
    lay.close()


@pytest.mark.parametrize("H,F,rows", [(256, 192, 21), (1728, 768, 26), (2880, 2880, 40)])
def test_rows_per_expert_from_which_the_fp16_kernel_takes_over(gpu_lib, port, H, F, rows):
    """The last batch of the block-scaled kernel and the first of the other, one expert: the images hold the one, and the
    results of both are the checker's."""
    sh = synth.tiny(seed=367, E=1, k=1, H=H, F=F, T=rows, has_bias=True)
    h, Wg, rb, ex = cases.layer_inputs(sh)
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    for n, path in ((rows - 1, 1), (rows, 2)):
        out, ro = lay.forward(h[:n])
        assert lay.timings()["path"] == path
        want, _ = port.moe_layer(h[:n], Wg, rb, ex, 1, sh.act, nthreads=8, router_out=ro)
        mx, mr = cases.err_stats(out, want)
        assert mx <= cases.MAX_ABS_OVER_RMS and mr <= cases.MEAN_REL, (mx, mr)
    lay.close()
