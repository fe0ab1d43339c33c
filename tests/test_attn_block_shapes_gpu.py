"""dg_attn_block over layers of different KV-head counts and canvases in one context: the projections' activations grow
with the widest of them, and what is kept for them (buffers, tensor maps) must follow."""
import pytest
import torch

from diffgemma_b200 import capi
from diffgemma_b200.step_attn import AttnBlock, AttnLayer, Context, KvCache
from tests import util
from tests.test_attn_block_gpu import _weights

pytestmark = pytest.mark.gpu

LAYERS = [dict(n_kv_heads=2, canvas=206), dict(n_kv_heads=8, canvas=80, window=512, mask_mode=capi.MASK_WINDOW_UNIFORM),
          dict(n_kv_heads=16, canvas=33), dict(n_kv_heads=2, canvas=256)]


def _step(ctx, lk, seed):
    layer = AttnLayer(n_q_heads=16, rope_theta=1e4, **lk)
    w = _weights(layer, 512, seed=seed, v_from_k=False)
    case = util.make_case(layer, 300, seed=seed)
    kv = KvCache(ctx, layer, 300 + layer.canvas)
    kv.load_prefix(case["kp"].cuda(), case["vp"].cuda(), 0)
    h = torch.randn(layer.canvas, 512, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).cuda()
    blk = AttnBlock(ctx, layer, **{k: t.cuda() for k, t in w.items()})
    out = blk.step(kv, 300, h).clone()
    ctx.synchronize()
    assert ctx.device_status()[0] == 0
    kv.close()
    return out.cpu()


def test_one_context_over_several_layers():
    alone = []
    for i, lk in enumerate(LAYERS):
        ctx = Context(0)
        alone.append(_step(ctx, lk, 40 + i))
        ctx.close()
    ctx = Context(0)
    for i, lk in enumerate(LAYERS):
        assert torch.equal(_step(ctx, lk, 40 + i), alone[i]), lk
    ctx.close()
