"""Saved sessions and raw appends: the one-launch copy between a token-major tensor and the cache against the strided
copies that host memory takes, and the vectorised stage 1 against the element-wise kernel that tensors off 16-byte
boundaries take.  Both pairs are the same values, so every comparison is of bits."""
import pytest
import torch

from diffgemma_b200 import capi
from diffgemma_b200.step_attn import AttnLayer, CanvasAttention, KvCache

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _randn(seed, *shape):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(*shape, generator=g).to(torch.bfloat16)


def _same(a, b):
    return torch.equal(a.cpu().view(torch.int16), b.cpu().view(torch.int16))


def _off_by_one(t):
    """The same values two bytes past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)
    out = buf[1:].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 16 == 2
    return out


@pytest.mark.parametrize("Hkv,D,n,pos0,ring", [
    (2, 512, 1, 0, None),          # one token
    (8, 256, 1023, 130, None),     # a count that no block of the copy divides
    (3, 80, 77, 5, None),          # rows of ten 16-byte chunks
    (8, 256, 700, 1800, 2048),     # the run wraps around the end of the ring
    (2, 256, 3000, 17, 2048),      # longer than the ring: only the last 2,048 positions are kept
])
def test_device_copy_equals_host_copy(ctx, Hkv, D, n, pos0, ring):
    layer = AttnLayer(n_q_heads=Hkv, n_kv_heads=Hkv, head_dim=D, rotary_dim=D, window=512, mask_mode=capi.MASK_WINDOW_UNIFORM)
    make = (lambda: KvCache(ctx, layer, ring_slots=ring)) if ring else (lambda: KvCache(ctx, layer, pos0 + n + 3))
    k, v = _randn(1, n, Hkv, D), _randn(2, n, Hkv, D)
    kept = min(n, ring) if ring else n
    a, b = make(), make()
    a.load_prefix(k.to(DEV), v.to(DEV), pos0)
    b.load_prefix(k, v, pos0)
    for kv in (a, b):
        got_k, got_v = kv.read(pos0 + n - kept, kept)
        assert _same(got_k, k[n - kept:]) and _same(got_v, v[n - kept:])
        if ring:
            whole_k, whole_v = kv.read(0, ring)          # slots outside the run are untouched
            gone = torch.ones(ring, dtype=torch.bool)
            gone[(torch.arange(pos0 + n - kept, pos0 + n) % ring)] = False
            assert not whole_k.cpu()[gone].any() and not whole_v.cpu()[gone].any()
        else:
            assert not kv.read(pos0 + n, 3)[0].any() and (pos0 == 0 or not kv.read(0, pos0)[1].any())
    # read into host memory and off a 16-byte boundary: the strided copies
    out = torch.empty(2, kept, Hkv, D, dtype=torch.bfloat16)
    capi.check(ctx.lib.dg_kv_read(a.h, out[0].data_ptr(), out[1].data_ptr(), pos0 + n - kept, kept), "dg_kv_read")
    assert _same(out[0], k[n - kept:]) and _same(out[1], v[n - kept:])
    c = make()
    c.load_prefix(_off_by_one(k), _off_by_one(v), pos0)
    assert _same(c.read(pos0 + n - kept, kept)[0], k[n - kept:])
    for kv in (a, b, c):
        kv.close()


@pytest.mark.parametrize("lk,n,pos0,write_end", [
    (dict(n_kv_heads=2, head_dim=512, rotary_dim=128, rope_theta=1e6, v_norm=1, rope_pairing=capi.ROPE_PROPORTIONAL), 1, 0, None),
    (dict(n_kv_heads=2, head_dim=512, rotary_dim=128, rope_theta=1e6, v_norm=1, rope_pairing=capi.ROPE_PROPORTIONAL), 1003, 131000, None),
    (dict(n_kv_heads=1, head_dim=512, rotary_dim=512, rope_theta=1e6), 6, 40, None),          # four tokens a CTA, ragged
    (dict(n_kv_heads=8, head_dim=256, rope_theta=1e4), 257, 999, 1100),                        # a padded chunk tail
    (dict(n_kv_heads=16, head_dim=256, rotary_dim=64, rope_theta=1e4), 33, 7, None),           # a partial rotation, split half
    (dict(n_kv_heads=2, head_dim=256, rotary_dim=0, rope_theta=1e4), 10, 3, None),             # none
])
@pytest.mark.parametrize("weights", [False, True])
def test_append_of_aligned_tensors_writes_the_same_bits(ctx, lk, n, pos0, write_end, weights):
    layer = AttnLayer(n_q_heads=16, **lk)
    H, D = layer.n_kv_heads, layer.head_dim
    k, v = _randn(3, n, H, D).to(DEV), _randn(4, n, H, D).to(DEV)
    kw = (1 + 0.1 * _randn(5, D)).to(torch.bfloat16).to(DEV) if weights else None
    a, b = KvCache(ctx, layer, pos0 + n), KvCache(ctx, layer, pos0 + n)
    a.append(k, v, pos0, kw, write_end)
    b.append(_off_by_one(k), _off_by_one(v), pos0, kw, write_end)
    for x, y in zip(a.read(0, pos0 + n), b.read(0, pos0 + n)):
        assert _same(x, y)
    assert a.read(pos0, 1)[0].any() and (write_end is None or not a.read(write_end, pos0 + n - write_end)[0].any())
    a.close()
    b.close()


@pytest.mark.parametrize("lk", [
    dict(n_kv_heads=2, head_dim=512, rotary_dim=128, rope_theta=1e6, v_norm=1, rope_pairing=capi.ROPE_PROPORTIONAL, canvas=37),
    dict(n_kv_heads=8, head_dim=256, rope_theta=1e4, canvas=256),
])
def test_stage_one_in_place_writes_the_same_bits(ctx, lk):
    layer = AttnLayer(n_q_heads=16, **lk)
    C, D, P = layer.canvas, layer.head_dim, 501
    x = [_randn(6 + i, C, h, D).to(DEV) for i, h in enumerate((16, layer.n_kv_heads, layer.n_kv_heads))]
    w = [(1 + 0.1 * _randn(9 + i, D)).to(torch.bfloat16).to(DEV) for i in range(2)]
    att = CanvasAttention(ctx, layer)
    a, b = KvCache(ctx, layer, P + C), KvCache(ctx, layer, P + C)
    aligned, shifted = [t.clone() for t in x], [_off_by_one(t) for t in x]
    att.qk_rope_kv(a, P, *aligned, *w)
    att.qk_rope_kv(b, P, *shifted, *w)
    ctx.synchronize()
    for t, u in zip(aligned + list(a.read(P, C)), shifted + list(b.read(P, C))):
        assert _same(t, u)
    assert not _same(aligned[0], x[0])
    a.close()
    b.close()


@pytest.mark.parametrize("hd,Hkv,n", [
    (256, 16, 128), (256, 16, 129),      # both sides of 4,096 vectors: four groups of eight a token, one CTA a token
    (256, 5, 7), (256, 9, 40),           # ten and eighteen vectors a token: two groups of five, three of six
    (256, 1, 2049), (512, 3, 1024), (512, 3, 1025), (512, 11, 3),
])
def test_append_groups_write_the_same_bits(ctx, hd, Hkv, n):
    layer = AttnLayer(n_q_heads=Hkv, n_kv_heads=Hkv, head_dim=hd, rotary_dim=hd // 2, rope_theta=1e5, v_norm=1)
    k, v, kw = _randn(11, n, Hkv, hd).to(DEV), _randn(12, n, Hkv, hd).to(DEV), (1 + 0.1 * _randn(13, hd)).to(torch.bfloat16).to(DEV)
    a, b = KvCache(ctx, layer, 77 + n), KvCache(ctx, layer, 77 + n)
    a.append(k, v, 77, kw)
    b.append(_off_by_one(k), _off_by_one(v), 77, kw)
    for x, y in zip(a.read(0, 77 + n), b.read(0, 77 + n)):
        assert _same(x, y) and x[77:].any() and not x[:77].any()
    a.close()
    b.close()


@pytest.mark.parametrize("hd,Hkv,canvas", [(256, 2, 17), (256, 8, 128), (256, 8, 129), (512, 2, 256)])
def test_stage_one_groups_write_the_table(ctx, hd, Hkv, canvas):
    """The first step at new positions: one group of a token writes its row of the RoPE table, the steps after it read it."""
    layer = AttnLayer(n_kv_heads=Hkv, head_dim=hd, rotary_dim=hd, rope_theta=1e4, canvas=canvas)
    q, k, v = _randn(14, 1, canvas, 16, hd).to(DEV), _randn(15, 1, canvas, Hkv, hd).to(DEV), _randn(16, 1, canvas, Hkv, hd).to(DEV)
    kv, att = KvCache(ctx, layer, 300 + canvas), CanvasAttention(ctx, layer)
    kv.load_prefix(_randn(17, 300, Hkv, hd), _randn(18, 300, Hkv, hd))
    first = att.denoise([kv], [300], q, k, v).clone()
    rows = [t.clone() for t in kv.read(300, canvas)]
    again = att.denoise([kv], [300], q, k, v)
    assert _same(first, again) and all(_same(x, y) for x, y in zip(rows, kv.read(300, canvas)))
    kv.close()
