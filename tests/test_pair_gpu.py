"""The fp16 tensor-core kernel of MXFP4 layers (CTA pairs) where its tiles, steps and tensor-memory plans end, against the CPU
restatement of the reference."""
import numpy as np
import pytest
import torch

from coalsack_b200 import MoeLayer, PATH_TILE, synth
from tests import cases

pytestmark = pytest.mark.gpu

MANY = 4128  # features: 33 tiles of gate/up, so that a pair walks several items


def row_tiles(rows):
    """Rows of the row tiles that the plan makes of the experts' rows: up to 256, two to four of an expert equally tall."""
    out = []
    for r in rows:
        n = -(-r // 256)
        per = min(256, (-(-r // n) + 31) // 32 * 32) if 2 <= n <= 4 else 256
        out += [min(per, r - at) for at in range(0, r, per)]
    return out


def contested(rows, weight_tiles, pairs):
    """How often a pair goes from an item to one whose accumulators do not fit beside it: the next item's MMAs then wait for the
    far columns.  (Columns: two slots of 64 for weights from 161 rows on, three from 129, else four.)"""
    mma = [max(32, (r + 31) // 32 * 32) for r in row_tiles(rows)]
    top = max(mma)
    columns = 512 - 64 * (4 if top <= 128 else 3 if top <= 160 else 2)
    items = [m for m in mma for _ in range(weight_tiles)]
    return sum(a + b > columns for a, b in zip(items, items[pairs:]))


@pytest.mark.parametrize("H,F,rows,bias,act,contests", [
    (32, 64, [1, 5], True, 0, False),                   # one k-tile per item: steps of one, dequantisers that skip whole items
    (64, 96, [33, 0, 31], False, 1, False),             # one and two k-tiles; an expert without rows
    (192, 320, [129, 128, 1], True, 0, False),          # odd k-tiles; a tile past 128 rows: three slots
    (192, 160, [32, 64, 96, 127], False, 1, False),     # 128 columns at most: four slots, eight stages
    (288, 352, [160, 161, 3], True, 1, False),          # the first tile of two slots
    (256, 288, [192, 193, 17], False, 0, False),
    (64, MANY, [160, 192, 160, 192, 160, 192], False, 0, False),  # the last accumulators that fit beside each other ...
    (64, MANY, [193, 192, 193, 192, 193, 192], False, 0, True),   # ... and the first that do not
    (128, MANY, [256, 225, 1, 256, 224, 256, 100, 255], True, 0, True),  # ... item after item, in every size
    (64, MANY, [257, 300, 513, 700], False, 1, True),   # several tiles per expert
    (32, MANY, [256] * 6, True, 1, True),               # items of one k-tile, all contested
    (128, MANY, [128] * 8, True, 1, False),             # nothing contested
])
def test_edges(gpu_lib, port, H, F, rows, bias, act, contests):
    T = sum(rows)
    sh = synth.tiny(seed=500 + T, E=len(rows), k=1, H=H, F=F, T=T, has_bias=bias, act=act)
    h, Wg, rb, ex = cases.layer_inputs(sh)
    route = np.ones((T, 1, 2), np.float32)
    route[:, 0, 0] = np.random.default_rng(T).permutation(np.repeat(np.arange(len(rows)), rows))
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    assert (contested(rows, -(-F // 128), pairs) > 0) == contests
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    lay.set_path(PATH_TILE)
    # (on device buffers: the host entry point cuts a batch into passes of lower tiles)
    d_h, d_route, d_out = torch.from_numpy(h).cuda(), torch.from_numpy(route).cuda(), torch.empty(T, H, device="cuda")
    torch.cuda.synchronize()

    def forward():
        d_out.zero_()
        torch.cuda.synchronize()
        lay.forward_dev(d_h, T, d_out, d_router_in=d_route)
        lay.sync()
        return d_out.cpu().numpy()

    out = forward()
    assert list(lay.counters()[0]) == list(rows)  # one launch for all of them
    want, _ = port.moe_layer(h, Wg, rb, ex, 1, act, nthreads=8, router_out=route)
    mx, mr = cases.err_stats(out, want)
    assert mx <= cases.MAX_ABS_OVER_RMS and mr <= cases.MEAN_REL, (mx, mr)
    for _ in range(3):  # an item's values do not depend on what ran beside it
        assert np.array_equal(out, forward())
    lay.close()
