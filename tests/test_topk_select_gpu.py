"""Selection of dg_attn_denoise_topk where its lists are at their limits: bounds below every visible key, keys that
cluster in few groups, more keys than the lists hold, key counts around the tiles of the score kernel; and the plane of
scores where it goes through several passes."""
import numpy as np
import pytest
import torch

from diffgemma_b200 import capi
from diffgemma_b200.step_attn import AttnLayer, CanvasAttention, Context, KvCache
from oracle import attn_oracle as ao
from tests import util
from tests.test_topk_gpu import _oracle, _run

pytestmark = pytest.mark.gpu

G256 = dict(n_q_heads=16, n_kv_heads=2, head_dim=256, canvas=256, rope_theta=1e6)
FULL = dict(n_q_heads=16, n_kv_heads=2, head_dim=512, canvas=256, rotary_dim=128, rope_theta=1e6, v_norm=1,
            rope_pairing=capi.ROPE_PROPORTIONAL)


def _check(ctx, case, **kcfg):
    got = _run(ctx, case, **kcfg)
    ref, gap = _oracle(case, return_gap=True, **kcfg)
    mx, mean, ties = ao.topk_errors(got, ref, gap)
    assert np.isfinite(got).all() and mx <= util.MAX_ABS_TOL and mean <= util.MEAN_ABS_TOL and ties <= 0.02, (mx, mean, ties)
    assert ctx.device_status()[0] == 0
    assert np.array_equal(got, _run(ctx, case, **kcfg))


@pytest.mark.parametrize("lk,P,kcfg", [
    (dict(G256, canvas=1), 0, dict(k_fixed=1, k_div=0)),               # one row, one key
    (dict(G256, canvas=3), 252, dict(k_fixed=16, k_div=0)),            # 255 keys: as many groups as kept keys
    (dict(G256, canvas=16), 240, dict(k_fixed=15, k_div=0)),           # 256 keys: one whole tile, one more group than kept keys
    (dict(G256, canvas=33), 224, dict(k_fixed=17, k_div=0)),           # 257 keys, rows that end inside a 128-row tile
    (dict(G256, n_kv_heads=16, canvas=40), 1000, dict(k_fixed=1024, k_div=0)),    # one query head per KV head; nearly all keys kept
    (dict(G256, n_kv_heads=1, canvas=64), 5000, dict(k_fixed=1024, k_div=0)),     # sixteen per KV head; fewer groups than kept keys
    (dict(FULL, canvas=65), 4033, dict(k_div=8, k_min=1, k_max=512)),
    (dict(FULL, canvas=20, window=300, mask_mode=capi.MASK_WINDOW_PER_ROW), 3000, dict(k_fixed=128, k_div=0)),   # more kept keys than groups in sight
])
def test_edges(ctx, lk, P, kcfg):
    _check(ctx, util.make_case(AttnLayer(**lk), P, seed=P + 3), **kcfg)


@pytest.mark.parametrize("run,k", [(16, 300), (300, 300), (64, 64)])
def test_clustered_keys(ctx, run, k):
    """Prefix keys that come in runs around one direction: the winners fill whole groups, and more keys than the lists of
    a warp hold reach the bound."""
    case = util.make_case(AttnLayer(**G256), 6000, seed=run)
    kp = util.t2f(case["kp"])
    rng = np.random.default_rng(run)
    near = kp[np.arange(len(kp)) // run * run] + 0.05 * rng.standard_normal(kp.shape).astype(np.float32)
    case["kp"] = util.f2t(near)
    _check(ctx, case, k_fixed=k, k_div=0)


def test_scores_are_no_further_from_64_bits(ctx):
    """Selected and weighted by the tensor cores' fp32 scores: against the same path in 64 bits the output error is that
    of its own rounding to bf16 (2^-9 of a value at most) plus that of P and the sums in fp32, below it."""
    layer = AttnLayer(**dict(FULL, canvas=32))
    case = util.make_case(layer, 5000, seed=12)
    got = _run(ctx, case, k_fixed=200, k_div=0).astype(np.float64)
    f = lambda n: util.t2f(case[n])
    d = case["desc"]
    qn, kn, vn = ao.qk_rope_kv(f("q"), f("kc"), f("vc"), None, None, d, 5000)
    K = np.concatenate([f("kp"), kn]).astype(np.float64)
    V = np.concatenate([f("vp"), vn]).astype(np.float64)
    worst = 0.0
    for h in range(16):
        s = qn[:, h].astype(np.float64) @ K[:, h // 8].T
        for i in range(32):
            order = np.argsort(-s[i], kind="stable")
            if (s[i, order[199]] - s[i, order[200]]) < 5e-6 * abs(s[i, order[199]]):
                continue
            t = order[:200]
            p = np.exp((s[i, t] - s[i, t].max()) * d.softmax_scale)
            ref = (p[:, None] * V[t, h // 8]).sum(0) / p.sum()
            worst = max(worst, float((np.abs(got[i, h] - ref) / np.maximum(np.abs(ref), 1e-2)).max()))
    # stage 1 rounds Q and the canvas K / V to bf16 on both sides in the same way up to one bf16 step of a few elements
    # (2^-8 of one of 512 products, a relative 1e-4 of a probability); half a bf16 step of the output is 2^-8 of its
    # leading bit at worst
    assert worst <= 2.0 ** -8 + 4e-3, worst


def _randn(seed, *shape):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").to(torch.bfloat16)


def test_shorter_range_is_capturable_after_a_longer_one():
    """30,000 keys go through the plane in two passes, 18,400 fill it in one: that call then finds its scratch in place."""
    ctx = Context(0)
    layer = AttnLayer(**G256)
    kv, att = KvCache(ctx, layer, 30000), CanvasAttention(ctx, layer)
    kv.load_prefix(_randn(1, 29744, 2, 256), _randn(2, 29744, 2, 256))
    q, k, v = _randn(3, 256, 16, 256), _randn(4, 256, 2, 256), _randn(5, 256, 2, 256)
    att.denoise_topk(kv, 29744, q, k, v)
    out = torch.empty_like(q)
    ctx.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=ctx.torch_stream):
        att.denoise_topk(kv, 18144, q, k, v, out=out)
    want = att.denoise_topk(kv, 18144, q, k, v)
    with torch.cuda.stream(ctx.torch_stream):
        out.zero_()
        g.replay()
    ctx.synchronize()
    assert out.any() and torch.equal(out, want) and ctx.device_status()[0] == 0
    del g
    ctx.close()


@pytest.mark.parametrize("lk,n_pass", [
    (dict(G256, n_kv_heads=8, canvas=250), 1),     # 16 row pairs, every other one ragged, in passes of 6, 6 and 4; a head alone: one
    (dict(FULL, canvas=256), 2),                   # the same passes; a head alone: two of 4
])
def test_passes_over_the_plane(ctx, lk, n_pass):
    """All heads in one call against a call per KV head: the same rows in other passes, so the same bits."""
    layer = AttnLayer(**lk)
    P, C, H, D, G = 42100, layer.canvas, layer.n_kv_heads, layer.head_dim, 16 // layer.n_kv_heads
    kp, vp = _randn(6, P, H, D), _randn(7, P, H, D)
    q, k, v = _randn(8, C, 16, D), _randn(9, C, H, D), _randn(10, C, H, D)
    kv = KvCache(ctx, layer, P + C)
    kv.load_prefix(kp, vp)
    got = CanvasAttention(ctx, layer).denoise_topk(kv, P, q, k, v)
    ctx.synchronize()
    assert ctx.last_launch_count == 1 + 2 * 3
    kv.close()
    one = AttnLayer(**dict(lk, n_q_heads=G, n_kv_heads=1))
    for h in range(H):
        kv = KvCache(ctx, one, P + C)
        kv.load_prefix(kp[:, h:h + 1].contiguous(), vp[:, h:h + 1].contiguous())
        want = CanvasAttention(ctx, one).denoise_topk(kv, P, q[:, h * G:(h + 1) * G].contiguous(), k[:, h:h + 1].contiguous(),
                                                      v[:, h:h + 1].contiguous())
        ctx.synchronize()
        assert ctx.last_launch_count == 1 + 2 * n_pass
        assert want.any() and torch.equal(got[:, h * G:(h + 1) * G], want), f"KV head {h}"
        kv.close()
    assert ctx.device_status()[0] == 0
