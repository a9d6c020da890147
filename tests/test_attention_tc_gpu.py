"""Prompt attention on the tcgen05 kernel at the key and value widths beside 128 x 128, against 64-bit torch."""
import math

import pytest
import torch

from volta_engine_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


def _want(q, k, v, pos, window, scale, gate=None):
    """q [n, nq, dk], k [ctx, nkv, dk], v [ctx, nkv, dv] of one sequence, 64 bits."""
    G = q.shape[1] // k.shape[1]
    s = torch.einsum("nhd,chd->nhc", q.double(), k.double().repeat_interleave(G, 1)) * scale
    key = torch.arange(k.shape[0], device=q.device)
    ok = key[None] <= pos[:, None]
    if window:
        ok &= key[None] > (pos - window)[:, None]
    p = torch.softmax(s.masked_fill(~ok[:, None], -math.inf), -1)
    o = torch.einsum("nhc,chd->nhd", p, v.double().repeat_interleave(G, 1))
    return o if gate is None else o * torch.sigmoid(gate.double()).reshape(o.shape)


def _err(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("hd", [128, 256])
@pytest.mark.parametrize("nq,nkv,start,n,window,gated,peak", [
    (2, 2, 0, 1, 0, False, 1.0), (16, 2, 0, 40, 0, False, 1.0), (24, 4, 63, 130, 0, True, 1.0), (16, 16, 600, 300, 0, False, 6.0),
    (32, 4, 500, 260, 192, True, 1.0), (128, 1, 190, 5, 0, False, 1.0), (8, 1, 3000, 600, 0, False, 3.0)])
def test_prompt_attention_pages_streams_and_maxima(hd, nq, nkv, start, n, window, gated, peak):
    """One page to many, one key-value head to as many as query heads, a window with a gate, two sequences in a launch, scores whose maximum
    moves by more than the lazy limit (``peak``). P is rounded to bf16 in front of the second product: 2^-9 a term, and the output once."""
    g = torch.Generator().manual_seed(n)
    maxp = (start + n + 63) // 64
    pages = 2 * maxp + 1
    table = (torch.randperm(pages - 1, generator=g) + 1).int().reshape(2, maxp).cuda()
    kp = (torch.randn(pages, nkv, 64, hd, generator=g) * peak).to(torch.bfloat16).cuda()
    vp = torch.randn(pages, nkv, 64, hd, generator=g).to(torch.bfloat16).cuda()
    half = n // 2
    slots = [1] * half + [0] * (n - half)
    starts = [start] * half + [start // 2] * (n - half)
    pos = torch.tensor([s + (i if i < half else i - half) for i, s in enumerate(starts)], dtype=torch.int32).cuda()
    q = torch.randn(n, (nq + 2 * nkv) * hd, generator=g).to(torch.bfloat16).cuda()
    gate = torch.randn(n, nq * hd, generator=g).to(torch.bfloat16).cuda() if gated else None
    tiles = K.make_prefill_tiles(slots, nq // nkv, "cuda")
    slot = torch.tensor(slots, dtype=torch.int32).cuda()
    got = K.attention(q, pos, slot, table, kp, vp, nq, nkv, hd, 1 / 16, tiles=tiles, window=window, gate=gate).reshape(n, nq, hd)
    for lo, hi, sl in ((0, half, 1), (half, n, 0)):
        if hi > lo:
            k = kp[table[sl].long()].transpose(1, 2).reshape(-1, nkv, hd)
            v = vp[table[sl].long()].transpose(1, 2).reshape(-1, nkv, hd)
            want = _want(q[lo:hi, :nq * hd].reshape(-1, nq, hd), k, v, pos[lo:hi], window, 1 / 16, None if gate is None else gate[lo:hi])
            assert _err(got[lo:hi], want) < 2 ** -8 + 2 ** -9
    assert K.check_status(torch.device("cuda")) == 0


@pytest.mark.parametrize("heads,start,n", [(1, 0, 1), (3, 0, 64), (5, 200, 129), (16, 37, 300), (32, 0, 1900)])
def test_latent_prompt_attention_keys_of_192(heads, start, n):
    """Keys and values expanded from the latent rows, then attention at 192 / 128 columns; the context ends inside a page."""
    from volta_engine_b200._lib import call, ptr
    g = torch.Generator().manual_seed(n)
    npages = (start + n + 63) // 64
    up = torch.randn(npages * 64, heads * 256, generator=g).to(torch.bfloat16).cuda()
    lat = torch.randn(npages * 64, 576, generator=g).to(torch.bfloat16).cuda()
    kp = torch.empty(npages, heads, 64, 192, dtype=torch.bfloat16, device="cuda")
    vp = torch.empty(npages, heads, 64, 128, dtype=torch.bfloat16, device="cuda")
    call("mla_expand_kv", "ppppiiii", ptr(up), ptr(lat), ptr(kp), ptr(vp), npages * 64, heads, 128, 128)
    u = up.reshape(-1, heads, 256)
    k = torch.cat([u[..., :128], lat[:, None, 512:].expand(-1, heads, -1)], -1)
    v = u[..., 128:]
    assert torch.equal(kp.transpose(1, 2).reshape(-1, heads, 192), k) and torch.equal(vp.transpose(1, 2).reshape(-1, heads, 128), v)
    q = torch.randn(n, heads * 192, generator=g).to(torch.bfloat16).cuda()
    pos = torch.arange(start, start + n, dtype=torch.int32).cuda()
    slot = torch.zeros(n, dtype=torch.int32, device="cuda")
    table = torch.arange(npages, dtype=torch.int32, device="cuda").reshape(1, npages)
    tf, tc, nt = K.make_prefill_tiles([0] * n, 1, "cuda", 128, False)
    out = torch.empty(n, heads * 128, dtype=torch.bfloat16, device="cuda")
    call("attention_k192_v128", "plplppppipipplifp", ptr(q), q.stride(0), ptr(out), out.stride(0), ptr(pos), ptr(slot), ptr(tf), ptr(tc), nt,
         ptr(table), npages, ptr(kp), ptr(vp), npages, heads, 0.07, ptr(K.status_word(q.device)))
    assert _err(out.reshape(n, heads, 128), _want(q.reshape(n, heads, 192), k, v, pos, 0, 0.07)) < 2 ** -8 + 2 ** -9
    assert K.check_status(torch.device("cuda")) == 0
