"""The work that the engine's speed is measured on: prompt portions, decode steps and verify blocks through ``Engine``, the call
that the scheduler makes, on the shapes of the repository's own model configurations with a few of their layers.

A case names a shape (``model``), what is run (``do``) and the sizes:

  prefill   one prompt of ``tokens`` rows in portions of at most 2048 rows, as the scheduler feeds them
  step      one step of ``rows`` rows: decode rows of ``rows`` streams with ``context`` cached tokens each, or, where ``streams``
            is 1, a block of ``rows`` rows behind the context of one stream (verification of drafted tokens)
  request   a prompt of ``tokens`` rows and ``new`` decode steps of one stream behind it

Outputs: the logits of the last forward and the caches and states that the pass wrote. ``exact`` is the same decoder in 64 bits
over the dequantised weights.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

import volta_engine_b200
from volta_engine_b200.models.dense import DenseConfig, DenseModel
from volta_engine_b200.models.hybrid import HybridConfig, HybridModel
from volta_engine_b200.models.mla import MLAConfig, MLAModel
from volta_engine_b200.models.moe import MoEConfig, MoEModel
from volta_engine_b200.ops.moe_gguf import GGUFExpertBank, parse_expert_quant
from volta_engine_b200.runtime.engine import Engine
from volta_engine_b200.runtime.kv_cache import PagedKVCache

PORTION = 2048
DEV = "cuda"


# ---------------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: a decode step of a small assistant model held as Q8_0, bound by launches
        dict(name="small_q8_step", model="small_q8", do="step", rows=1, streams=1, context=191),
        # one user's chat with a 27B-class dense model behind a long document, NVFP4
        dict(name="dense_nvfp4_step", model="dense_nvfp4", do="step", rows=1, streams=1, context=16384),
        # the prompt in front of it
        dict(name="dense_nvfp4_prefill", model="dense_nvfp4", do="prefill", tokens=3001),
        # the same model from a Q4_K file, four streams
        dict(name="dense_q4k_step", model="dense_q4k", do="step", rows=4, streams=4, context=1500),
        # 512 experts as trellis codes: one user, sixteen users, a prompt
        dict(name="moe_exl3_step", model="moe_exl3", do="step", rows=1, streams=1, context=8192),
        dict(name="moe_exl3_streams", model="moe_exl3", do="step", rows=16, streams=16, context=700),
        dict(name="moe_exl3_prefill", model="moe_exl3", do="prefill", tokens=2500),
        # latent attention: four rows (three drafted tokens behind the last one) verified at 16K
        dict(name="mla_exl3_verify", model="mla_exl3", do="step", rows=4, streams=1, context=16384),
        # a large model served from GGUF blocks: a decode step of eight streams, a prompt
        dict(name="mla_gguf_streams", model="mla_gguf", do="step", rows=8, streams=8, context=2000),
        dict(name="mla_gguf_prefill", model="mla_gguf", do="prefill", tokens=1900),
        # linear attention beside full attention: a prompt, and a short request as an agent sends it
        dict(name="hybrid_prefill", model="hybrid", do="prefill", tokens=4000),
        dict(name="hybrid_request", model="hybrid", do="request", tokens=150, new=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# per shape: largest prompt, largest context of a single stream
RANGES = {"small_q8": (200, 191), "dense_nvfp4": (3001, 16384), "dense_q4k": (3001, 8192), "moe_exl3": (2500, 16384),
          "mla_exl3": (1900, 16384), "mla_gguf": (1900, 8192), "hybrid": (4000, 8192)}


def draw(rng):
    model = rng.choice(sorted(RANGES))
    tokens, context = RANGES[model]
    do = rng.choice(["prefill", "request"] if model == "hybrid" else ["prefill", "step", "step"])
    if do == "prefill":
        return dict(model=model, do=do, tokens=_log(rng, 40, tokens))
    if do == "request":
        return dict(model=model, do=do, tokens=_log(rng, 20, 600), new=rng.randint(2, 8))
    rows = rng.choice([1, 1, 2, 3, 4, 5, 8, 11, 16])
    if rng.random() < 0.5:
        return dict(model=model, do=do, rows=rows, streams=1, context=_log(rng, 30, context - 16))
    return dict(model=model, do=do, rows=rows, streams=rows, context=_log(rng, 30, min(2000, context)))


def tolerance(case):
    # bf16 activations between the layers: against 64 bits the logits, caches and states were 0.005 to 0.008 off on the shapes with
    # routed experts (whose residual stream is large beside a layer's output), 0.01 to 0.021 on the others
    return {"rel": 0.02 if case["model"].startswith(("moe", "mla")) else 0.03, "max": 0.6}


# ---------------------------------------------------------------------------------------------------------------- the models
def _config(name):
    if name == "small_q8":
        return DenseConfig(n_layers=4, hidden=512, n_q=8, n_kv=2, head_dim=64, ffn=1408, vocab=32000, quant="gguf_q8_0")
    if name == "dense_nvfp4":
        cfg = DenseConfig.baseline_27b()
        cfg.n_layers = 4
    elif name == "dense_q4k":
        cfg = DenseConfig.baseline_27b()
        cfg.n_layers, cfg.quant, cfg.vocab = 3, "gguf_q4_k", 32000
    elif name == "moe_exl3":
        cfg = MoEConfig.baseline_moe()
        cfg.n_layers, cfg.expert_quant = 4, "exl3_4"
    elif name == "mla_exl3":
        cfg = MLAConfig.baseline_mla_mtp()
        cfg.n_layers, cfg.mtp_layers, cfg.expert_quant = 4, 0, "exl3_3"
    elif name == "mla_gguf":
        cfg = MLAConfig.baseline_dsv3()
        cfg.n_layers, cfg.first_dense_layers, cfg.quant, cfg.expert_quant = 3, 1, "gguf_q8_0", "gguf_iq1_m"
    else:
        cfg = HybridConfig.dense_27b()
        cfg.n_layers = 4
    return cfg


def _model(name, seed):
    cfg = _config(name)
    kinds = {"moe_exl3": MoEModel, "mla_exl3": MLAModel, "mla_gguf": MLAModel, "hybrid": HybridModel}
    m = kinds.get(name, DenseModel)(cfg, DEV)
    m.init_random(seed=seed)
    if name == "mla_gguf":
        for li, L in enumerate(m.layers):
            if not L.dense_ffn:          # block scales that put the weights at the spread of the other matrices
                L.bank = None
                L.bank = GGUFExpertBank.random(cfg.n_experts, cfg.expert_ffn, cfg.hidden, *parse_expert_quant(cfg.expert_quant),
                                               seed=seed * 1009 + li, device=DEV, amp=0.004)
    if isinstance(m, MoEModel) and name != "hybrid":
        # a trained router is sure of its choice: every token has a topic that its residual stream carries, and the experts of
        # the topic stand out by more than rounding moves a score
        g = torch.Generator(device=DEV).manual_seed(seed + 77)
        E, k, H = cfg.n_experts, cfg.top_k, cfg.hidden
        topics = E // k
        T = (torch.randint(0, 2, (topics, H), generator=g, device=DEV) * 2 - 1).float()
        of = torch.arange(topics * k, device=DEV).reshape(k, topics)          # a topic's experts lie in k groups of experts
        m.embed.copy_(torch.randn(m.embed.shape, generator=g, device=DEV))
        m.embed.add_((2.0 * T)[torch.arange(m.embed.shape[0], device=DEV) % topics].to(m.embed.dtype))
        for L in m.layers:
            if not L.dense_ffn:
                w = L.router.weight
                if cfg.n_group > 1:       # k experts in topk_group groups
                    per, gs = k // cfg.topk_group, E // cfg.n_group
                    first = torch.randint(0, cfg.n_group, (topics,), generator=g, device=DEV)
                    place = torch.randint(0, gs - per, (topics, cfg.topk_group), generator=g, device=DEV)
                    grp = (first[:, None] + torch.arange(cfg.topk_group, device=DEV)) % cfg.n_group
                    ids = ((grp * gs + place)[..., None] + torch.arange(per, device=DEV)).reshape(topics, k)
                else:
                    ids = of.t()
                add = torch.zeros(w.shape, device=DEV)
                for j in range(k):
                    add.index_add_(0, ids[:, j], T * (16.0 / H))
                w.add_(add.to(w.dtype))
    return m, cfg


def _ids(case, seed, n):
    g = torch.Generator().manual_seed(seed + 5)
    return torch.randint(0, 32000, (n,), generator=g).tolist()


def prepare(case, seed):
    m, cfg = _model(case["model"], seed)
    do = case["do"]
    slots = case["streams"] if do == "step" else 1
    per = case["context"] + case["rows"] // case["streams"] + 2 if do == "step" else case["tokens"] + case.get("new", 0) + 2
    pages = slots * ((per + 63) // 64 + 1) + 1
    if case["model"].startswith("mla"):
        kv = PagedKVCache(cfg.n_layers, 1, 576, pages, slots, per + 64, DEV, v_head_dim=8)
    elif case["model"] == "hybrid":
        kv = PagedKVCache(m.kv_layers, m.nkv, cfg.head_dim, pages, slots, per + 64, DEV)
    else:
        kv = PagedKVCache(cfg.n_layers, m.nkv, cfg.head_dim, pages, slots, per + 64, DEV)
    s = {"model": m, "cfg": cfg, "kv": kv, "engine": Engine(m, kv, prefill_chunk=PORTION, feedback=False), "do": do}
    if do == "step":
        g = torch.Generator(device=DEV).manual_seed(seed + 3)     # what earlier steps left in the cache
        kv.k.normal_(generator=g)
        kv.v.normal_(generator=g)
        n = case["rows"]
        s["ids"] = _ids(case, seed, n)
        one = case["streams"] == 1
        s["slots"] = [0] * n if one else list(range(n))
        # streams have contexts of their own lengths
        s["pos"] = [case["context"] + r for r in range(n)] if one else [max(1, case["context"] - 37 * r) for r in range(n)]
        for slot, p in zip(s["slots"], s["pos"]):
            kv.reserve(slot, p + 2)
    else:
        s["ids"] = _ids(case, seed, case["tokens"])
        s["more"] = _ids(case, seed + 1, case.get("new", 0))
    return s


def run(s):
    eng = s["engine"]
    if s["do"] == "step":
        eng.step(s["ids"], s["pos"], s["slots"])
    else:
        n = len(s["ids"])
        for p in range(0, n, PORTION):
            eng.prefill_rows(0, s["ids"][p:p + PORTION], p, p + PORTION >= n)
        for i, t in enumerate(s["more"]):
            eng.step([t], [n + i], [0])
    out = {"logits": eng.row_logits, "k": s["kv"].k}
    if s["kv"].v_head_dim > 8:
        out["v"] = s["kv"].v
    st = [x for x in getattr(s["model"], "gdn_states", None) or [] if x is not None]
    if st:
        out["state"] = [x.rec for x in st]
    return out


# ---------------------------------------------------------------------------------------------------------------- the work
def _bits(cfg):
    dense = {"nvfp4": 4.5, "gguf_q8_0": 8.5, "gguf_q4_k": 4.5}[cfg.quant]
    expert = {"exl3_4": 4.0, "exl3_3": 3.0, "gguf_iq1_m": 1.75, "nvfp4": 4.5}[cfg.expert_quant] if hasattr(cfg, "expert_quant") else 0.0
    return dense, expert


def work(case):
    """Weights that the rows need once, the cached tokens that they see once, the rows' own cache entries and the logits."""
    name = case["model"]
    cfg = _config(name)
    dense_bits, expert_bits = _bits(cfg)
    H = cfg.hidden
    step = case["do"] == "step"
    forwards = [(case["rows"], case["context"], case["streams"])] if step else \
        [(min(PORTION, case["tokens"] - p), p, 1) for p in range(0, case["tokens"], PORTION)] + \
        [(1, case["tokens"] + i, 1) for i in range(case.get("new", 0))]
    mla = name.startswith("mla")
    nbytes = flops = 0.0
    for fi, (n, ctx, streams) in enumerate(forwards):
        for li in range(cfg.n_layers):
            full = name != "hybrid" or (li + 1) % cfg.full_interval == 0
            keys = ctx + (0 if streams > 1 else n / 2)
            if mla:
                hd = cfg.n_q * (cfg.qk_nope + cfg.v_head_dim)
                w = H * (cfg.q_lora_rank + 576) + cfg.q_lora_rank * cfg.n_q * (cfg.qk_nope + cfg.qk_rope) + cfg.n_q * cfg.v_head_dim * H
                nbytes += hd * 512 * 2 + 576 * 2 * (ctx * max(1, streams) + n)
                # scores and values of every key, at the cheaper of the two ways to read a latent row
                up = min(2 * n * hd * 512 + 2 * n * keys * cfg.n_q * (576 + 512), 2 * (ctx + n) * hd * 512 + 2 * n * keys * cfg.n_q * (192 + 128))
                flops += up
            elif full:
                w = H * (cfg.n_q + 2 * cfg.n_kv) * cfg.head_dim + cfg.n_q * cfg.head_dim * H
                if name == "hybrid":
                    w += H * cfg.n_q * cfg.head_dim
                nbytes += 2 * 2 * cfg.n_kv * cfg.head_dim * (ctx * max(1, streams) + n)
                flops += 4 * n * keys * cfg.n_q * cfg.head_dim
            else:
                C = 2 * cfg.gdn_k_heads * cfg.gdn_dk + cfg.gdn_v_heads * cfg.gdn_dv
                w = H * (C + cfg.gdn_v_heads * cfg.gdn_dv + 2 * cfg.gdn_v_heads) + cfg.gdn_v_heads * cfg.gdn_dv * H
                nbytes += 2 * 4 * cfg.gdn_v_heads * cfg.gdn_dk * cfg.gdn_dv
                flops += 7 * n * cfg.gdn_v_heads * cfg.gdn_dk * cfg.gdn_dv
            nbytes += w * dense_bits / 8
            flops += 2 * n * w
            if name in ("moe_exl3", "mla_exl3", "mla_gguf") and li >= cfg.first_dense_layers:
                topics = cfg.n_experts // cfg.top_k
                seen = cfg.top_k * topics * (1 - (1 - 1 / topics) ** n)
                one, sh = 3 * H * cfg.expert_ffn, 3 * H * cfg.shared_ffn
                nbytes += seen * one * expert_bits / 8 + sh * dense_bits / 8 + cfg.n_experts * H * 2
                flops += 2 * n * (cfg.top_k * one + sh + cfg.n_experts * H)
            else:
                nbytes += 3 * H * cfg.ffn * dense_bits / 8
                flops += 2 * n * 3 * H * cfg.ffn
        last = step or fi == len(forwards) - 1 or n == 1
        if last:
            rows = n if step else 1
            head_bits = dense_bits if name in ("small_q8", "dense_nvfp4", "dense_q4k") else 16
            nbytes += H * cfg.vocab * head_bits / 8 + 4 * rows * cfg.vocab
            flops += 2 * rows * H * cfg.vocab
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------------------------------------------- 64 bits
def _f16(b):
    """[..., 2] bytes -> the number that they hold"""
    return b.contiguous().view(torch.float16)[..., 0].double()


def _nvfp4(packed, scales, gscale):
    lut = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6, 0, -0.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64, device=packed.device)
    v = torch.stack((packed & 15, packed >> 4), -1).flatten(-2)
    v = lut[v.int()].reshape(*scales.shape, 16)
    return (v * (scales.view(torch.float8_e4m3fn).double() * gscale)[..., None]).flatten(-2)


def _q8_0(raw, K):
    b = raw.reshape(-1, K // 32, 34)
    return (b[..., 2:].view(torch.int8).double() * _f16(b[..., :2])[..., None]).flatten(-2)


def _q4_k(raw, K):
    b = raw.reshape(-1, K // 256, 144)
    s = b[..., 4:16].int()
    scale = torch.cat([s[..., 0:4] & 63, (s[..., 8:12] & 15) | (s[..., 0:4] >> 6 << 4)], -1)
    low = torch.cat([s[..., 4:8] & 63, (s[..., 8:12] >> 4) | (s[..., 4:8] >> 6 << 4)], -1)
    q = b[..., 16:].reshape(*b.shape[:2], 4, 32)
    q = torch.stack([q & 15, q >> 4], 3).reshape(*b.shape[:2], 8, 32).double()
    d, dmin = _f16(b[..., 0:2])[..., None], _f16(b[..., 2:4])[..., None]
    return (q * (d * scale)[..., None] - (dmin * low)[..., None]).reshape(-1, K)


def _iq1_m(raw, K):
    path = os.path.join(os.path.dirname(volta_engine_b200.__file__), "quant", "data", "iq_grids.bin")
    grid = torch.from_numpy(np.fromfile(path, dtype=np.int8)[17536:].reshape(2048, 8).copy()).to(raw.device).double()
    b = raw.reshape(-1, K // 256, 56)
    lo, qh = b[..., :32].int().reshape(*b.shape[:2], 16, 2), b[..., 32:48].int()
    sc = b[..., 48:56].int()
    sc = sc[..., 0::2] | sc[..., 1::2] << 8
    d = (sc[..., 0] >> 12) | (sc[..., 1] >> 8 & 0xF0) | (sc[..., 2] >> 4 & 0xF00) | (sc[..., 3] & 0xF000)
    d = torch.where(d >= 32768, d - 65536, d).to(torch.int16)[..., None].view(torch.float16)[..., 0].double()
    at = torch.arange(16, device=raw.device)                  # groups of 16 weights: four 3-bit scales in a word
    dl = d[..., None] * (2 * (sc[..., at // 4] >> (3 * (at % 4)) & 7) + 1)
    idx = torch.stack([lo[..., 0] | (qh << 8 & 0x700), lo[..., 1] | (qh << 4 & 0x700)], -1)
    shift = torch.where(torch.stack([qh & 8, qh & 128], -1) != 0, -0.125, 0.125).double()
    return ((grid[idx] + shift[..., None]) * dl[..., None, None]).reshape(-1, K)


def _linear(lin):
    """The weights [out, in] of a linear as the model holds them."""
    if hasattr(lin, "raw"):
        return (_q8_0 if lin.ggml_type == 8 else _q4_k)(lin.raw, lin.in_features)
    if hasattr(lin, "packed"):
        w = _nvfp4(lin.packed, lin.scales, lin.gscale)
        if getattr(lin, "gated", False):                      # tiles of 64 gate and 64 up rows
            w = w.reshape(-1, 2, 64, w.shape[1]).transpose(0, 1).reshape(-1, w.shape[1])
        return w
    return lin.weight.double()


_H128 = None


def _had(x):
    global _H128
    if _H128 is None:
        h = torch.ones(1, 1, dtype=torch.float64, device=x.device)
        while h.shape[0] < 128:
            h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)])
        _H128 = h / math.sqrt(128)
    return (x.reshape(-1, 128) @ _H128).reshape(x.shape)


def _exl3(codes, bits):
    """Trellis codes [K/16, N/16, 16 bits] -> the rotated weights [K, N]; sum-of-bytes codebook."""
    c = codes.long() & 0xFFFF
    words = c[..., 0::2] | c[..., 1::2] << 16
    p = torch.arange(256, device=codes.device)
    start = (p * bits + bits - 16) % (256 * bits)
    w0, off = start // 32, start % 32
    both = words[..., w0] << 16 | words[..., (w0 + 1) % words.shape[-1]] >> 16       # 48 bits from the window's first word on
    x = (both >> (32 - off) & 0xFFFF) * 0x83DCD12D & 0xFFFFFFFF
    s = (x & 255) + (x >> 8 & 255) + (x >> 16 & 255) + (x >> 24)
    a, b = np.array([0x1EEE, 0xC931], dtype=np.uint16).view(np.float16).astype(np.float64)
    v = ((1024 + s).double() * a + b).half().double()
    lane, i = p // 8, p % 8
    row, col = (lane & 3) * 2 + (i & 1) + 8 * (i >> 1 & 1), 2 * (lane // 8 + 4 * (i >> 2)) + (lane >> 2 & 1)
    t = torch.empty(*codes.shape[:2], 16, 16, dtype=torch.float64, device=codes.device)
    t[:, :, row, col] = v
    return t.permute(0, 2, 1, 3).reshape(codes.shape[0] * 16, codes.shape[1] * 16)


def _expert(bank, e, x, cfg):
    I = cfg.expert_ffn
    if hasattr(bank, "gate"):
        s, n = bank.s, bank.bits

        def lin(v, codes, su, sv):
            return _had(_had(v * s[su][e].double()) @ _exl3(codes[e], n)) * s[sv][e].double()
        a = torch.nn.functional.silu(lin(x, bank.gate, "g_suh", "g_svh")) * lin(x, bank.up, "u_suh", "u_svh")
        return lin(a, bank.down, "d_suh", "d_svh")
    gu = x @ _iq1_m(bank.gu_raw[e], cfg.hidden).t()
    return (torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]) @ _iq1_m(bank.dn_raw[e], I).t()


def _norm(x, w, cfg):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + cfg.rms_eps) * (w.double() + cfg.norm_bias)


def _rope(v, pos, rot, theta):
    """v [rows, heads, width]: the first ``rot`` columns turn, in two halves."""
    half = rot // 2
    ang = pos[:, None, None].double() * theta ** (-torch.arange(half, device=v.device).double() / half)
    a, b = v[..., :half], v[..., half:rot]
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin(), v[..., rot:]], -1)


def _softmax_rows(q, k, v, pos, scale):
    """q [n, w], k [t, w], v [t, w2]; a row sees the keys up to its own position."""
    s = (q @ k.t()) * scale
    s.masked_fill_(torch.arange(k.shape[0], device=q.device)[None] > pos[:, None], float("-inf"))
    return torch.softmax(s, -1) @ v


def _delta_net(x, g, d, eps):
    """The gated delta rule over a whole sequence: outputs and the last state."""
    n, C, nv = x.shape[0], d.conv_dim, d.n_v
    p = x @ _linear(g["in_proj"]).t()
    raw = torch.nn.functional.pad(p[:, :C], (0, 0, d.conv_k - 1, 0))
    cw = g["conv_w"].double()
    u = torch.nn.functional.silu(sum(raw[j:j + n] * cw[:, j] for j in range(d.conv_k)))
    q, k = u[:, :d.n_k * d.dk].reshape(n, d.n_k, d.dk), u[:, d.n_k * d.dk:2 * d.n_k * d.dk].reshape(n, d.n_k, d.dk)
    v = u[:, 2 * d.n_k * d.dk:].reshape(n, nv, d.dv)
    q, k = (t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = (t.repeat_interleave(nv // d.n_k, 1) for t in (q * d.dk ** -0.5, k))
    z, rest = p[:, C:C + nv * d.dv].reshape(n, nv, d.dv), p[:, C + nv * d.dv:]
    beta = torch.sigmoid(rest[:, :nv])
    decay = torch.exp(-torch.exp(g["A_log"].double()) * torch.nn.functional.softplus(rest[:, nv:2 * nv] + g["dt_bias"].double()))
    S = torch.zeros(nv, d.dk, d.dv, dtype=torch.float64, device=x.device)
    o = torch.empty_like(v)
    for i in range(n):
        S.mul_(decay[i][:, None, None])
        kk = k[i][:, None]
        S.baddbmm_(k[i][..., None], (v[i][:, None] - kk @ S) * beta[i][:, None, None])
        o[i] = (q[i][:, None] @ S)[:, 0]
    o = o * torch.rsqrt((o * o).mean(-1, keepdim=True) + eps) * g["norm_w"].double() * torch.nn.functional.silu(z)
    return o.reshape(n, -1) @ _linear(g["out_proj"]).t(), S


def _feed_forward(L, x, cfg):
    def swiglu(v, gu, dn):
        a = v @ _linear(gu).t()
        I = a.shape[1] // 2
        return (torch.nn.functional.silu(a[:, :I]) * a[:, I:]) @ _linear(dn).t()
    if getattr(L, "bank", None) is None:
        return swiglu(x, L.gate_up, L.down)
    lg = x @ _linear(L.router).t()
    score = torch.sigmoid(lg) if cfg.router == "sigmoid" else lg
    pick = score
    if cfg.n_group > 1:
        grp = score.reshape(len(x), cfg.n_group, -1)
        keep = grp.topk(2, -1).values.sum(-1).topk(cfg.topk_group, -1).indices
        mask = torch.zeros(grp.shape[:2], dtype=torch.bool, device=x.device).scatter_(1, keep, True)
        pick = grp.masked_fill(~mask[..., None], float("-inf")).reshape(score.shape)
    ids = pick.topk(cfg.top_k, -1).indices
    w = score.gather(1, ids)
    w = (w / (w.sum(-1, keepdim=True) + 1e-9) if cfg.router == "sigmoid" else torch.softmax(w, -1)) * cfg.router_scale
    y = swiglu(x, L.shared_gu, L.shared_dn)
    for e in ids.unique().tolist():
        r, j = (ids == e).nonzero(as_tuple=True)
        y.index_add_(0, r, _expert(L.bank, e, x[r], cfg) * w[r, j][:, None])
    return y


def exact(case, seed):
    s = prepare(case, seed)
    m, cfg, kv = s["model"], s["cfg"], s["kv"]
    if s["do"] == "step":
        ids, where = s["ids"], list(zip(s["slots"], s["pos"]))
    else:
        ids = s["ids"] + s["more"]
        where = [(0, p) for p in range(len(ids))]
        kv.reserve(0, len(ids) + 1)
    pos = torch.tensor([p for _, p in where], device=DEV)
    segments = []                                              # (slot, first row, rows): rows behind one another
    for r, (slot, p) in enumerate(where):
        if segments and segments[-1][0] == slot:
            segments[-1][2] += 1
        else:
            segments.append([slot, r, 1])
    table = kv.host_table.long()
    page = torch.stack([table[slot, p // 64] for slot, p in where]).to(DEV)
    kc, vc = kv.k.double(), kv.v.double()

    def cached(pool, slot, n):
        pages = table[slot, :(n + 63) // 64].to(DEV)
        return pool[pages].transpose(1, 2).reshape(-1, pool.shape[1], pool.shape[3])[:n]          # [tokens, heads, width]
    h = m.embed[torch.tensor(ids, device=DEV)].double()
    n, hd, state, full = len(ids), cfg.head_dim, [], 0
    for L in m.layers:
        x = _norm(h, L.attn_norm, cfg)
        if getattr(L, "gdn", None) is not None:
            o, S = _delta_net(x, L.gdn, m.dims, cfg.rms_eps)
            state.append(S[None])
        elif getattr(L, "qkv_a", None) is not None:
            a, ql = x @ _linear(L.qkv_a).t(), cfg.q_lora_rank
            q = (_norm(a[:, :ql], L.q_a_norm, cfg) @ _linear(L.q_b).t()).reshape(n, cfg.n_q, -1)
            q_rot = _rope(q[..., cfg.qk_nope:], pos, 64, cfg.rope_theta)
            q = torch.cat([torch.einsum("nhd,hdc->nhc", q[..., :cfg.qk_nope], L.w_uk.double()), q_rot], -1)
            kc[full][page, 0, pos % 64] = torch.cat([_norm(a[:, ql:ql + 512], L.kv_a_norm, cfg),
                                                     _rope(a[:, None, ql + 512:ql + 576], pos, 64, cfg.rope_theta)[:, 0]], -1)
            o = torch.empty(n, cfg.n_q, 512, dtype=torch.float64, device=DEV)
            for slot, r, c in segments:
                lat = cached(kc[full], slot, where[r][1] + c)[:, 0]
                for i in range(cfg.n_q):
                    o[r:r + c, i] = _softmax_rows(q[r:r + c, i], lat, lat[:, :512], pos[r:r + c], m.scale)
            o = torch.einsum("nhc,hvc->nhv", o, L.w_uv.double()).reshape(n, -1) @ _linear(L.o_proj).t()
            full += 1
        else:
            a = (x @ _linear(L.qkv).t()).reshape(n, -1, hd)
            q, k, v = a.split([cfg.n_q, cfg.n_kv, cfg.n_kv], 1)
            if cfg.qk_norm:
                q, k = _norm(q, L.q_norm, cfg), _norm(k, L.k_norm, cfg)
            rot = cfg.rot_dim or hd
            q = _rope(q, pos, rot, cfg.rope_theta)
            kc[full][page, :, pos % 64], vc[full][page, :, pos % 64] = _rope(k, pos, rot, cfg.rope_theta), v
            o = torch.empty_like(q)
            for slot, r, c in segments:
                ks, vs = cached(kc[full], slot, where[r][1] + c), cached(vc[full], slot, where[r][1] + c)
                for i in range(cfg.n_q):
                    j = i // (cfg.n_q // cfg.n_kv)
                    o[r:r + c, i] = _softmax_rows(q[r:r + c, i], ks[:, j], vs[:, j], pos[r:r + c], m.scale)
            o = o.reshape(n, -1)
            if getattr(L, "gate_proj", None) is not None:
                o = o * torch.sigmoid(x @ _linear(L.gate_proj).t())
            o = o @ _linear(L.o_proj).t()
            full += 1
        h = h + o
        h = h + _feed_forward(L, _norm(h, L.ffn_norm, cfg), cfg)
    x = _norm(h if s["do"] == "step" else h[-1:], m.final_norm, cfg)
    out = {"logits": x @ _linear(m.lm_head).t(), "k": kc}
    if kv.v_head_dim > 8:
        out["v"] = vc
    if state:
        out["state"] = state
    return out
