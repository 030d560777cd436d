"""The fp16 tensor-core kernel of MXFP4 layers (CTA pairs) where its tiles, steps and tensor-memory plans end, against the CPU
restatement of the reference."""
import numpy as np
import pytest

from coalsack_b200 import MoeLayer, PATH_TILE, synth
from tests import cases

pytestmark = pytest.mark.gpu

MANY = 4128  # features: 33 tiles of gate/up, so that a pair walks several items


@pytest.mark.parametrize("H,F,rows,bias,act", [
    (32, 64, [1, 5], True, 0),                   # one k-tile per item: steps of one, dequantisers that skip whole items
    (64, 96, [33, 0, 31], False, 1),             # one and two k-tiles; an expert without rows
    (192, 320, [129, 128, 1], True, 0),          # odd k-tiles; a tile past 128 rows: three slots
    (192, 160, [32, 64, 96, 127], False, 1),     # 128 columns at most: four slots, eight stages
    (288, 352, [160, 161, 3], True, 1),          # the first tile of two slots
    (256, 288, [192, 193, 17], False, 0),        # the first accumulators that contest columns
    (128, MANY, [256, 225, 1, 256, 224, 256, 100, 255], True, 0),  # ... item after item, in every size
    (64, MANY, [257, 300, 513, 700], False, 1),  # several tiles per expert
    (128, MANY, [128] * 8, True, 1),             # nothing contested
])
def test_edges(gpu_lib, port, H, F, rows, bias, act):
    T = sum(rows)
    sh = synth.tiny(seed=500 + T, E=len(rows), k=1, H=H, F=F, T=T, has_bias=bias, act=act)
    h, Wg, rb, ex = cases.layer_inputs(sh)
    route = np.ones((T, 1, 2), np.float32)
    route[:, 0, 0] = np.random.default_rng(T).permutation(np.repeat(np.arange(len(rows)), rows))
    lay = MoeLayer.from_shape(sh)
    lay.set_router(Wg, rb)
    lay.load_experts(ex)
    lay.set_path(PATH_TILE)
    out, _ = lay.forward(h, router_out=route)
    assert lay.timings()["path"] == PATH_TILE
    want, _ = port.moe_layer(h, Wg, rb, ex, 1, act, nthreads=8, router_out=route)
    mx, mr = cases.err_stats(out, want)
    assert mx <= cases.MAX_ABS_OVER_RMS and mr <= cases.MEAN_REL, (mx, mr)
    for _ in range(3):  # an item's values do not depend on what ran beside it
        again, _ = lay.forward(h, router_out=route)
        assert np.array_equal(out, again)
    lay.close()
