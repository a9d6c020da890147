"""Prompt attention on the tcgen05 kernel at heads of 128 and 256 columns, against 64-bit torch."""
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


@pytest.mark.parametrize("hd", [128, 256])
def test_prompt_rows_whose_window_lies_behind_their_key_limit(hd):
    """A tile without a page to read writes zeros, as the 64-row kernel does; its neighbours, in the same launch, see their keys."""
    n, nq, nkv, window = 70, 4, 2, 64
    g = torch.Generator().manual_seed(hd)
    kp, vp = (torch.randn(20, nkv, 64, hd, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    table = torch.arange(20, dtype=torch.int32).reshape(1, 20).cuda()
    pos = torch.arange(1000, 1000 + n, dtype=torch.int32).cuda()
    key_end = pos.clone()
    key_end[:64] = 10                              # G = 2: the first tile of 64 tokens sees nothing, the second one all
    q = torch.randn(n, nq * hd, generator=g).to(torch.bfloat16).cuda()
    slot = torch.zeros(n, dtype=torch.int32).cuda()
    out = []
    for wide in (True, False):
        tiles = K.make_prefill_tiles([0] * n, nq // nkv, "cuda", wide=wide)
        out.append(K.attention(q, pos, slot, table, kp, vp, nq, nkv, hd, 1 / 16, out=torch.full((n, nq * hd), 7.0, dtype=torch.bfloat16, device="cuda"),
                               tiles=tiles, window=window, key_end=key_end))
    assert not out[0][:64].any() and not out[1][:64].any()
    assert _err(out[0][64:], out[1][64:].double()) < 2 ** -7
    assert K.check_status(torch.device("cuda")) == 0


@pytest.mark.parametrize("nq,nkv,start,n,window,peak", [(24, 4, 0, 300, 0, 1.0), (16, 2, 200, 900, 0, 4.0), (8, 1, 1500, 300, 256, 3.0), (4, 4, 0, 700, 0, 8.0)])
def test_prompt_attention_of_256_columns_is_as_near_as_the_64_row_kernel(nq, nkv, start, n, window, peak):
    """Its probabilities are rounded from the same numbers, so its distance to 64 bits is the other kernel's but for the order of fp32 sums."""
    hd, g = 256, torch.Generator().manual_seed(n)
    maxp = (start + n + 63) // 64
    table = torch.arange(maxp, dtype=torch.int32).reshape(1, maxp).cuda()
    kp = (torch.randn(maxp, nkv, 64, hd, generator=g) * peak).to(torch.bfloat16).cuda()
    vp = torch.randn(maxp, nkv, 64, hd, generator=g).to(torch.bfloat16).cuda()
    pos = torch.arange(start, start + n, dtype=torch.int32).cuda()
    q = torch.randn(n, nq * hd, generator=g).to(torch.bfloat16).cuda()
    slot = torch.zeros(n, dtype=torch.int32).cuda()
    k, v = (t.transpose(1, 2).reshape(-1, nkv, hd) for t in (kp, vp))
    want = _want(q.reshape(n, nq, hd), k, v, pos, window, 1 / 16)
    far = []
    for wide in (True, False):
        tiles = K.make_prefill_tiles([0] * n, nq // nkv, "cuda", wide=wide)
        far.append(_err(K.attention(q, pos, slot, table, kp, vp, nq, nkv, hd, 1 / 16, tiles=tiles, window=window).reshape(n, nq, hd), want))
    assert far[0] < 1.005 * far[1], far
    assert K.check_status(torch.device("cuda")) == 0


@pytest.mark.parametrize("heads,npages,nope,vd", [(1, 1, 128, 128), (5, 3, 64, 72), (3, 2, 192, 256)])
def test_latent_keys_and_values_expanded_into_pages(heads, npages, nope, vd):
    """Bytes as they are, zeros behind the columns in use."""
    from volta_engine_b200._lib import call, ptr
    up = torch.randn(npages * 64, heads * (nope + vd)).to(torch.bfloat16).cuda()
    lat = torch.randn(npages * 64, 576).to(torch.bfloat16).cuda()
    k, v = (torch.full((npages, heads, 64, 256), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    call("mla_expand_kv", "ppppiiii", ptr(up), ptr(lat), ptr(k), ptr(v), npages * 64, heads, nope, vd)
    u = up.reshape(-1, heads, nope + vd)
    k, v = (t.transpose(1, 2).reshape(-1, heads, 256) for t in (k, v))
    assert torch.equal(k[..., :nope], u[..., :nope]) and torch.equal(v[..., :vd], u[..., nope:])
    assert torch.equal(k[..., nope:nope + 64], lat[:, None, 512:].expand(-1, heads, -1))
    assert not k[..., nope + 64:].any() and not v[..., vd:].any()
