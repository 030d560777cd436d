"""The block-scaled expert kernel (weights as MXFP4 operands, token rows as five E2M1 digits) where its tiles, records and
padding end, against the CPU restatement of the reference."""
import numpy as np
import pytest

from coalsack_b200 import MoeLayer, PATH_STREAM, synth
from tests import cases

pytestmark = pytest.mark.gpu

# A block's digits leave at most 2^-14.2 of its largest value (0.2 of what an fp16 operand leaves, in norm); two
# contractions and fp32 sums in another order stay well under 1e-3 of the output's RMS.
MX_MAX, MX_MEAN = 2e-3, 3e-4


@pytest.mark.parametrize("E,k,H,F,T,bias,act,wbf", [
    (2, 1, 32, 32, 1, False, 0, False),      # one block: half of the K = 64 step is padding, 32 of 128 rows exist
    (2, 2, 96, 160, 3, True, 1, False),      # odd block counts either way; 15 of 16 columns
    (1, 1, 128, 128, 48, True, 0, False),    # one full tile (240 columns), one whole record
    (1, 1, 160, 384, 49, True, 0, True),     # two even tiles; second half of a plain unit absent; routing weight first
    (1, 1, 256, 288, 22, False, 0, False),   # the last height with two accumulator pairs ...
    (1, 1, 256, 288, 23, False, 1, False),   # ... and the first with one
    (3, 2, 288, 352, 145, True, 0, False),   # several tiles per expert, uneven loads
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
