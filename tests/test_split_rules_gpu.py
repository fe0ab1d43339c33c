"""Key splits under a decoder bitmap (a cluster shares the merge of fp32 rows) and the launch shapes that the split and pair
rules choose: short key ranges with odd tile counts, several canvases of equal and unequal lengths, in-launch
appends of every unit size."""
import numpy as np
import pytest
import torch

from diffgemma_b200 import capi
from diffgemma_b200.step_attn import AttnLayer, CanvasAttention, KvCache
from tests import util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hkv,canvas,P", [(2, 256, 900), (8, 100, 333), (16, 17, 1200)])
def test_bitmap_splits(ctx, Hkv, canvas, P):
    layer = AttnLayer(n_kv_heads=Hkv, canvas=canvas, rope_theta=1e6)
    case = util.make_case(layer, P, seed=P)
    rng = np.random.default_rng(P)
    attend = rng.random((canvas, P + canvas)) < 0.4
    attend[:, :P // 3] = False
    attend[0] = False                                  # a row that sees nothing
    ref = util.run_oracle(case, attend=attend)
    kv, att = util.gpu_setup(ctx, case)
    a = torch.from_numpy(attend.astype(np.uint8)).cuda()
    try:
        for splits in (0, 1, 2, 3, 4, 8):
            ctx.set_splits(splits)
            got = util.t2f(att.denoise_bitmap(kv, P, util.dev(case, "q"), util.dev(case, "kc"), util.dev(case, "vc"), a))
            util.assert_close(got, ref, f"bitmap, {splits} splits")
            assert not got[0].any()
    finally:
        ctx.set_splits(0)
        kv.close()


@pytest.mark.parametrize("Hkv,canvas,P,batch", [
    (8, 256, 8229, 4),      # unsplit pairs, four heads per append unit
    (8, 200, 1100, 2),      # two canvases
    (2, 256, 770, 3),
    (8, 150, 2000, 1),      # an odd number of query tiles per KV head: no pairs
    (8, 100, 433, 1),       # a short range, unsplit
    (16, 33, 90, 1), (1, 64, 500, 1),
])
def test_automatic_launch_shapes(ctx, Hkv, canvas, P, batch):
    layer = AttnLayer(n_kv_heads=Hkv, canvas=canvas, rope_theta=1e4, window=1024, mask_mode=capi.MASK_WINDOW_PER_ROW)
    cases = [util.make_case(layer, P, seed=50 + b) for b in range(batch)]
    kvs = [util.gpu_setup(ctx, c)[0] for c in cases]
    att = CanvasAttention(ctx, layer)
    q, k, v = (torch.stack([c[n] for c in cases]).cuda() for n in ("q", "kc", "vc"))
    refs = [util.run_oracle(c) for c in cases]
    first = att.denoise(kvs, [P] * batch, q, k, v).clone()
    again = att.denoise(kvs, [P] * batch, q, k, v).clone()      # the append runs inside this launch
    ctx.synchronize()
    assert torch.equal(first, again) and ctx.device_status()[0] == 0
    for b in range(batch):
        util.assert_close(util.t2f(again[b]), refs[b], f"canvas {b}")
        kvs[b].close()


@pytest.mark.parametrize("Hkv,canvas,P,batch", [(8, 100, 333, 1), (8, 256, 500, 1), (2, 256, 200, 1), (2, 64, 700, 1), (8, 256, 600, 2),
                                                (1, 17, 100, 4)])
def test_short_ranges_keep_fp32_sums(ctx, Hkv, canvas, P, batch):
    """Up to six key tiles (seven for 64 query tiles) the automatic choice is one split, whose sums stay fp32 to the rounded
    output: the same bits as with one split forced."""
    layer = AttnLayer(n_kv_heads=Hkv, canvas=canvas, rope_theta=1e4, window=1024, mask_mode=capi.MASK_WINDOW_UNIFORM)
    cases = [util.make_case(layer, P, seed=90 + b) for b in range(batch)]
    kvs = [util.gpu_setup(ctx, c)[0] for c in cases]
    att = CanvasAttention(ctx, layer)
    q, k, v = (torch.stack([c[n] for c in cases]).cuda() for n in ("q", "kc", "vc"))
    got = att.denoise(kvs, [P] * batch, q, k, v).clone()
    try:
        ctx.set_splits(1)
        want = att.denoise(kvs, [P] * batch, q, k, v)
        ctx.synchronize()
    finally:
        ctx.set_splits(0)
    assert torch.equal(got, want) and ctx.device_status()[0] == 0
    for kv in kvs:
        kv.close()


@pytest.mark.parametrize("Hkv,canvas,mask,Ps", [
    (8, 256, capi.MASK_WINDOW_UNIFORM, (333, 5000, 5000, 5000)),      # 5 and 11 key tiles: both sides of where pairs begin to pay
    (8, 256, capi.MASK_WINDOW_UNIFORM, (2000, 600, 9000)),
    (2, 256, capi.MASK_NONE, (333, 2048)),
    (2, 256, capi.MASK_NONE, (500, 4000, 4000, 4000)),
    (2, 256, capi.MASK_NONE, (0, 700, 40, 4000, 260)),                # two launches of up to four
    (8, 256, capi.MASK_CAUSAL, (0, 1500)),                            # query tiles whose first split has no key tile
    (8, 256, capi.MASK_WINDOW_PER_ROW, (10, 3000)),
])
def test_unequal_canvases_share_a_launch(ctx, Hkv, canvas, mask, Ps):
    layer = AttnLayer(n_kv_heads=Hkv, canvas=canvas, rope_theta=1e4, window=1024 if mask else 0, mask_mode=mask)
    cases = [util.make_case(layer, P, seed=70 + b) for b, P in enumerate(Ps)]
    kvs = [util.gpu_setup(ctx, c)[0] for c in cases]
    att = CanvasAttention(ctx, layer)
    q, k, v = (torch.stack([c[n] for c in cases]).cuda() for n in ("q", "kc", "vc"))
    att.denoise(kvs, list(Ps), q, k, v)
    got = att.denoise(kvs, list(Ps), q, k, v)      # positions known: the appends run inside the attention launch
    ctx.synchronize()
    assert ctx.last_launch_count == (len(Ps) + 3) // 4 and ctx.device_status()[0] == 0
    for b, case in enumerate(cases):
        util.assert_close(util.t2f(got[b]), util.run_oracle(case), f"canvas {b}")
        kvs[b].close()
