"""fp16 weights on CTA pairs: row tiles, weight tiles and k-tiles where they end, the layer without clusters of two, and the
order of the weights in image files."""
import numpy as np
import pytest
import torch

from coalsack_b200 import CskError, MoeLayer, synth
from tests import cases

pytestmark = pytest.mark.gpu


def _layer(H, F, T, act=synth.STANDARD_SWIGLU, E=1, k=1, seed=31, bias=True):
    experts = [cases.dense_ffn_case(H=H, F=F, T=1, bias=bias, seed=seed + e)[1:] for e in range(E)]
    lay = MoeLayer(E, k, H, F, activation=act, has_bias=bias, max_tokens=T, weights_f16=True)
    for e, w in enumerate(experts):
        gw, uw, dw = w[:3]
        lay.load_expert_f16(e, uw, gw, dw, *((w[4], w[3], w[5]) if bias else ()))
    return lay, experts


EDGES = [
    (32, 32, 65),       # one k-tile, half of it padding; half of the features of a CTA's rows real, none of the other's
    (64, 96, 255), (64, 160, 256), (96, 128, 257),   # a row tile's last height, two even ones
    (192, 64, 97),      # both halves of a row tile ragged: 49 rows in one of 64
    (320, 288, 513), (2080, 32, 80),                 # three row tiles; more k-tiles than stages, of the lowest tiles too
    (512, 544, 160),
]


@pytest.mark.parametrize("H,F,T", EDGES)
def test_edges(gpu_lib, port, H, F, T):
    lay, ((gw, uw, dw, bg, bu, bd),) = _layer(H, F, T)
    hidden = np.random.default_rng(T).standard_normal((T, H)).astype(np.float32)
    out = lay.dense_forward(hidden)
    mx, mr = cases.err_stats(out, port.dense_ffn(hidden, gw, uw, dw, bg, bu, bd))
    assert mx <= cases.MAX_ABS_OVER_RMS and mr <= cases.MEAN_REL, (mx, mr)
    for _ in range(3):
        assert np.array_equal(lay.dense_forward(hidden), out)
    lay.close()


@pytest.mark.parametrize("clusters", [True, False])
def test_waits_run_out_and_the_handle_recovers(gpu_lib, clusters):
    """A copy role that issues nothing under a wait budget of 0.1 ms: the call reports it, the next one computes as before."""
    lay, _ = _layer(256, 192, 300)
    if not clusters:
        lay.debug_set(lay.DEBUG_NO_CLUSTERS, 1)
    hidden = np.random.default_rng(3).standard_normal((300, 256)).astype(np.float32)
    good = lay.dense_forward(hidden)
    try:
        lay.debug_set(lay.DEBUG_WAIT_BUDGET, 200_000)
        lay.debug_set(lay.DEBUG_STALL_TILE_PRODUCER, 1)
        with pytest.raises(CskError) as err:
            lay.dense_forward(hidden)
        assert err.value.code == -3 and "wait ran out" in str(err.value)
    finally:
        lay.debug_set(lay.DEBUG_WAIT_BUDGET, 2_000_000_000)
    assert np.array_equal(lay.dense_forward(hidden), good)
    lay.close()


@pytest.mark.parametrize("E,k,T", [(1, 1, 300), (3, 2, 700)])
def test_without_clusters_a_cta_takes_half_a_weight_tile(gpu_lib, E, k, T):
    """Every batch of more rows than the kernel for few of them takes goes to the tensor-core kernel's form without clusters."""
    H, F = 160, 288
    lay, _ = _layer(H, F, T, E=E, k=k, bias=False)
    rng = np.random.default_rng(5)
    lay.set_router((rng.standard_normal((E, H)) * 0.1).astype(np.float32), None)
    hidden = rng.standard_normal((T, H)).astype(np.float32)
    want, _ = lay.forward(hidden)
    lay.debug_set(lay.DEBUG_NO_CLUSTERS, 1)
    got, _ = lay.forward(hidden)
    # an activation may round to the next fp16 (2^-11 of it) where its two sums differ: one of 288 in a sum, 2e-3 of the rms at most
    assert np.abs(got - want).max() <= 2e-3 * want.std() and np.abs(got - want).mean() <= 1e-4 * want.std()
    lay.close()


@pytest.mark.parametrize("H,F,T", EDGES)
def test_edges_without_clusters(gpu_lib, port, H, F, T):
    lay, ((gw, uw, dw, bg, bu, bd),) = _layer(H, F, T)
    lay.debug_set(lay.DEBUG_NO_CLUSTERS, 1)
    hidden = np.random.default_rng(T).standard_normal((T, H)).astype(np.float32)
    out = lay.dense_forward(hidden)
    mx, mr = cases.err_stats(out, port.dense_ffn(hidden, gw, uw, dw, bg, bu, bd))
    assert mx <= cases.MAX_ABS_OVER_RMS and mr <= cases.MEAN_REL, (mx, mr)
    for _ in range(3):
        assert np.array_equal(lay.dense_forward(hidden), out)
    lay.close()


def test_received_rows_without_clusters(gpu_lib):
    """Rows of peers (here the layer's own), whose results go to their places through a map."""
    E, k, H, F, T = 3, 2, 160, 288, 200
    lay, _ = _layer(H, F, T, E=E, k=k, bias=False)
    rng = np.random.default_rng(6)
    lay.set_router((rng.standard_normal((E, H)) * 0.1).astype(np.float32), None)
    hidden = rng.standard_normal((T, H)).astype(np.float32)
    lay.debug_set(lay.DEBUG_NO_CLUSTERS, 1)
    want, _ = lay.forward(hidden)
    send = torch.zeros((T * k, lay.ep_row_pitch()), dtype=torch.float16, device="cuda")
    counts = torch.zeros(E, dtype=torch.int32, device="cuda")
    back, out = torch.zeros((T * k, H), device="cuda"), torch.empty((T, H), device="cuda")
    x = torch.from_numpy(hidden).cuda()
    torch.cuda.synchronize()
    lay.ep_dispatch_dev(x, T, send, counts)
    lay.ep_experts_dev(send, counts, 1, T * k, back)
    lay.ep_combine_dev(back, T, out)
    lay.sync()
    assert np.array_equal(out.cpu().numpy(), want)
    lay.close()


def test_image_files_keep_their_order(gpu_lib, tmp_path):
    """The gate rows of 128 features first, then their up rows, as before the device's order changed: 16-byte pieces at piece ^ (row & 7)."""
    H, F = 96, 160
    lay, ((gw, uw, dw, *_),) = _layer(H, F, 4)
    img = tmp_path / "w.img"
    lay.save_image(img)
    blob = np.fromfile(img, np.uint8)
    header = 8 + 8 * 4 + 7 * 8
    off_tgu = int(np.frombuffer(blob[8 + 32 + 24:8 + 32 + 32].tobytes(), np.uint64)[0])
    record = blob[header + 1:]  # (one expert: one flag)
    tile = record[off_tgu:off_tgu + 2 * 2 * 2 * 16384].view(np.float16).reshape(2, 2, 2, 128, 8, 8)  # [n_tile][k_tile][half][row][piece][8]
    for half, w in ((0, gw), (1, uw)):
        rows = np.zeros((256, 128), np.float16)
        rows[:F, :H] = w
        for r in (0, 17, 63, 64, 100, 127):
            for n in range(2):
                for kt in range(2):
                    got = tile[n, kt, half, r][np.arange(8) ^ (r & 7)].reshape(-1)
                    assert np.array_equal(got, rows[128 * n + r, 64 * kt:64 * kt + 64]), (half, n, kt, r)
    again, _ = _layer(H, F, 4, seed=77)
    again.load_image(img)
    hidden = np.random.default_rng(1).standard_normal((4, H)).astype(np.float32)
    assert np.array_equal(again.dense_forward(hidden), lay.dense_forward(hidden))
    lay.close()
    again.close()
