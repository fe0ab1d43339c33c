"""Decoder-bitmap calls at the edges of what the tensor kernels take: whatever they cannot take has to come out as the
general kernel computes it."""
import numpy as np
import pytest
import torch

from diffgemma_b200 import capi
from diffgemma_b200.step_attn import AttnLayer, CanvasAttention, Context, KvCache
from tests import util

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _layer(hd, canvas, **more):
    if hd == 512:
        return AttnLayer(n_kv_heads=2, head_dim=512, canvas=canvas, rotary_dim=128, rope_theta=1e6, v_norm=1,
                         rope_pairing=capi.ROPE_PROPORTIONAL, **more)
    return AttnLayer(n_kv_heads=2, canvas=canvas, rope_theta=1e6, **more)


def _case(hd, P, canvas, seed, **more):
    case = util.make_case(_layer(hd, canvas, **more), P, seed=seed, weights=True)
    seen = np.random.default_rng(seed).random((canvas, P + canvas)) < 0.6
    args = [util.dev(case, n) for n in ("q", "kc", "vc")] + [torch.from_numpy(seen.astype(np.uint8)).to(DEV)]
    return case, seen, args + [util.dev(case, "qw"), util.dev(case, "kw")]


def _general(ctx, att, kv, P, args):
    try:
        ctx.force_general(True)
        return att.denoise_bitmap(kv, P, *args).clone()
    finally:
        ctx.force_general(False)


def _off_by_one(t):
    """The same values two bytes past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)
    out = buf[1:].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 16 == 2
    return out


@pytest.mark.parametrize("hd", [256, 512])
@pytest.mark.parametrize("which", ["q", "k", "v", "qw", "kw", "out"])
def test_tensors_off_16_byte_boundaries(ctx, hd, which):
    P, canvas = 300, 40
    case, _, args = _case(hd, P, canvas, seed=hd + 1)
    kv, att = util.gpu_setup(ctx, case)
    want = _general(ctx, att, kv, P, args)
    cache = [t.clone() for t in kv.read(0, P + canvas)]
    kv.close()
    kv, att = util.gpu_setup(ctx, case)
    out = torch.empty_like(args[0])
    at = {"q": 0, "k": 1, "v": 2, "qw": 4, "kw": 5}
    if which == "out":
        out = _off_by_one(out)
    else:
        args[at[which]] = _off_by_one(args[at[which]])
    for step in range(2):       # the second step finds the positions' RoPE table in memory
        out.fill_(7.0)
        att.denoise_bitmap(kv, P, *args, out=out)
        ctx.synchronize()
        assert torch.equal(out, want), f"step {step}"
        for got, ref in zip(kv.read(0, P + canvas), cache):
            assert torch.equal(got, ref)
    kv.close()


@pytest.mark.parametrize("hd,P,canvas,splits", [(256, 300, 40, 0), (256, 1500, 100, 4), (256, 700, 256, 1), (256, 700, 33, 3),
                                                (512, 200, 17, 0), (512, 900, 100, 3)])
@pytest.mark.parametrize("bad", ["padding", "holes", "canvas", "visible"])
def test_keys_without_numbers(ctx, hd, P, canvas, splits, bad):
    """Infinite and NaN keys and values behind zero bits: hidden from all rows, or from some of them.  A row that sees none
    of them is the same as over finite keys (against the general kernel one bf16 step, 2^-7 of a value, and what the order of
    the sums leaves near zero); one that does is what the general kernel makes of it."""
    case, seen, args = _case(hd, P, canvas, seed=hd + P)
    if bad == "padding":
        where = np.arange(0, 130)               # a dead tile and the head of a live one
    elif bad == "canvas":
        where = P + np.arange(0, canvas, 5)
    else:
        where = np.array([3, 131, 140, P - 1])
    if bad == "visible":
        seen[:, where] = False
        seen[1::3, where[1]] = True
    else:
        seen[:, where] = False
    args[3] = torch.from_numpy(seen.astype(np.uint8)).to(DEV)
    kinds = torch.tensor([float("nan"), float("inf"), float("-inf")], dtype=torch.bfloat16, device=DEV)
    kv, att = util.gpu_setup(ctx, case)
    clean = _general(ctx, att, kv, P, args)
    if bad == "canvas":
        for j, t in enumerate(where):
            args[2][int(t) - P] = kinds[j % 3]
    else:
        k, v = case["kp"].to(DEV), case["vp"].to(DEV)
        for j, t in enumerate(where):
            v[int(t)] = kinds[j % 3]
            if bad != "visible":
                k[int(t), :, ::2] = kinds[(j + 1) % 3]
        kv.load_prefix(k, v, 0)
    want = _general(ctx, att, kv, P, args)
    blind = torch.from_numpy(~seen[:, where].any(axis=1)).to(DEV)
    assert torch.equal(want[blind], clean[blind])
    try:
        ctx.set_splits(splits)
        for _ in range(2):
            got = att.denoise_bitmap(kv, P, *args)
            ctx.synchronize()
            torch.testing.assert_close(got.float(), want.float(), rtol=2.0 ** -7, atol=2e-3, equal_nan=True)
    finally:
        ctx.set_splits(0)
    assert ctx.device_status()[0] == 0
    kv.close()


@pytest.mark.parametrize("hd", [256, 512])
def test_output_over_the_queries(ctx, hd):
    P, canvas = 300, 40
    case, _, args = _case(hd, P, canvas, seed=hd + 2)
    kv, att = util.gpu_setup(ctx, case)
    want = _general(ctx, att, kv, P, args)
    att.denoise_bitmap(kv, P, *args, out=args[0])
    ctx.synchronize()
    assert torch.equal(args[0], want)
    kv.close()


@pytest.mark.parametrize("P,canvas", [(600, 100), (2000, 256)])
def test_ring_positions_that_are_gone(ctx, P, canvas):
    """A bitmap on a ring may show positions that the ring no longer holds: they read what took their slots, the canvas of
    this very step among it, in the second step too, whose append runs inside the attention launch."""
    layer = AttnLayer(n_kv_heads=2, canvas=canvas, rope_theta=1e4, window=64, mask_mode=capi.MASK_WINDOW_UNIFORM)
    kv = KvCache(ctx, layer, ring_slots=512)
    att = CanvasAttention(ctx, layer)
    g = torch.Generator(device=DEV).manual_seed(P)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV).to(torch.bfloat16)
    kv.append(rn(P, 2, 256), rn(P, 2, 256), 0)
    seen = (torch.rand(canvas, P + canvas, generator=g, device=DEV) < 0.5).to(torch.uint8)
    for _ in range(3):
        args = rn(canvas, 16, 256), rn(canvas, 2, 256), rn(canvas, 2, 256), seen
        got = att.denoise_bitmap(kv, P, *args).clone()
        want = _general(ctx, att, kv, P, args)
        torch.testing.assert_close(got.float(), want.float(), rtol=2.0 ** -7, atol=2e-3)
    assert ctx.device_status()[0] == 0
    kv.close()


@pytest.mark.parametrize("hd", [256, 512])
def test_captured_before_any_scratch_exists(hd):
    """A bitmap call is recorded in a context that has run nothing yet, then the scratch grows under eager calls several
    times: the replay still works on memory of its own."""
    ctx = Context(0)
    P, canvas = 900, 40
    case, seen, args = _case(hd, P, canvas, seed=hd + 3)
    kv, att = util.gpu_setup(ctx, case)
    out = torch.empty_like(args[0])
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=ctx.torch_stream):
        att.denoise_bitmap(kv, P, *args, out=out)
    others = []
    for P2, canvas2 in ((1500, 100), (9000, 256)):
        c2, seen2, args2 = _case(hd, P2, canvas2, seed=P2)
        kv2, att2 = util.gpu_setup(ctx, c2)
        for splits in (0, 8):
            ctx.set_splits(splits)
            got = util.t2f(att2.denoise_bitmap(kv2, P2, *args2))
            util.assert_close(got, util.run_oracle(c2, attend=seen2), f"{P2} keys, {splits} splits")
        ctx.set_splits(0)
        others.append((att2, kv2, P2, args2))
    want = util.run_oracle(case, attend=seen)
    for att2, kv2, P2, args2 in others:
        att2.denoise_bitmap(kv2, P2, *args2)
        with torch.cuda.stream(ctx.torch_stream):
            out.zero_()
            g.replay()
        ctx.synchronize()
        util.assert_close(util.t2f(out), want, "replay")
    assert ctx.device_status()[0] == 0
    del g
    ctx.close()


@pytest.mark.parametrize("hd,heads", [(256, 4097), (512, 2049)])
def test_more_query_tiles_than_a_tensor_launch_takes(ctx, hd, heads):
    layer = AttnLayer(n_q_heads=heads, n_kv_heads=heads, head_dim=hd, canvas=1, rotary_dim=hd, rope_theta=1e6)
    kv, att = KvCache(ctx, layer, 101), CanvasAttention(ctx, layer)
    g = torch.Generator(device=DEV).manual_seed(hd)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV).to(torch.bfloat16)
    kv.append(rn(100, heads, hd), rn(100, heads, hd), 0)
    args = rn(1, heads, hd), rn(1, heads, hd), rn(1, heads, hd), (torch.rand(1, 101, generator=g, device=DEV) < 0.5).to(torch.uint8)
    want = _general(ctx, att, kv, 100, args)
    got = att.denoise_bitmap(kv, 100, *args)
    ctx.synchronize()
    assert want.any() and torch.equal(got, want)
    kv.close()


@pytest.mark.parametrize("hd,P,canvas,small", [(256, 0, 1, True), (256, 46, 18, True), (256, 47, 18, False), (256, 45, 19, False),
                                               (512, 14, 18, True), (512, 15, 18, False), (512, 13, 19, False)])
def test_small_calls(ctx, hd, P, canvas, small):
    """Both sides of the line below which the general kernel is the quicker one (64 keys of 256, two rows a multiprocessor)."""
    case, seen, args = _case(hd, P, canvas, seed=hd + P)
    kv, att = util.gpu_setup(ctx, case)
    want = _general(ctx, att, kv, P, args)
    ctx.kernel_timing(True, 4)       # counts the launches of the tensor kernels
    got = att.denoise_bitmap(kv, P, *args)
    launches = ctx.kernel_time()[1]
    ctx.kernel_timing(False)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert sms != 148 or launches == (0 if small else 1)
    if small:
        assert torch.equal(got, want)
    util.assert_close(util.t2f(got), util.run_oracle(case, attend=seen), "bitmap")
    kv.close()
