"""MLA attention (absorbed decode kernel, expanded prefill) and the MTP head against the fp32 CPU statement."""
import pytest
import torch

from volta_engine_b200.models.mla import MLAConfig, MLAModel
from volta_engine_b200.models.util import to_device
from volta_engine_b200.runtime.batch import BatchRows
from volta_engine_b200.runtime.kv_cache import PagedKVCache
from util import cos

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _kv(m, dev):
    return PagedKVCache(m.cfg.n_layers + m.cfg.mtp_layers, 1, 576, 24, 2, 1024, dev, v_head_dim=8)


@pytest.mark.parametrize("heads", [4, 20])
def test_mla_prefill_then_decode_matches_reference(heads):
    cfg = MLAConfig.tiny_mla(n_q=heads)
    mg = MLAModel(cfg, DEV).init_random(seed=5)
    mc = to_device(mg, "cpu")
    mg.ensure_workspace(16, 8)
    kvg, kvc = _kv(mg, DEV), _kv(mc, "cpu")
    prompt = torch.randint(0, cfg.vocab, (150,), generator=torch.Generator().manual_seed(2)).tolist()
    kvg.reserve(0, 256)
    kvc.reserve(0, 256)
    G = 1
    bg = BatchRows.make(prompt, list(range(150)), [0] * 150, DEV, "last", G, prefill=True)
    bc = BatchRows.make(prompt, list(range(150)), [0] * 150, "cpu", "last", G, prefill=True)
    lg, lc = mg.forward(bg, kvg), mc.forward(bc, kvc)
    assert cos(lg.cpu(), lc) > 0.995, "prefill logits"
    # latent cache rows written by both paths agree
    pg = kvg.k[0][kvg.host_table[0, 0].item(), 0, :64].float().cpu()
    pc = kvc.k[0][kvc.host_table[0, 0].item(), 0, :64].float()
    assert cos(pg, pc) > 0.999
    # decode / verify rows through the absorbed kernel, several split factors
    for nsplit in (1, 3):
        ids = [5, 9, 11]
        pos = [150, 151, 152]
        bg2 = BatchRows.make(ids, pos, [0] * 3, DEV, "all", G, nsplit=nsplit)
        bc2 = BatchRows.make(ids, pos, [0] * 3, "cpu", "all", G)
        lg2, lc2 = mg.forward(bg2, kvg), mc.forward(bc2, kvc)
        assert cos(lg2.cpu(), lc2) > 0.995, f"decode logits nsplit={nsplit}"
    from volta_engine_b200.ops import kernels as K
    assert K.check_status(DEV) == 0


def test_mtp_head_matches_reference():
    cfg = MLAConfig.tiny_mla()
    mg = MLAModel(cfg, DEV).init_random(seed=6)
    mc = to_device(mg, "cpu")
    mg.ensure_workspace(16, 8)
    kvg, kvc = _kv(mg, DEV), _kv(mc, "cpu")
    kvg.reserve(0, 64)
    kvc.reserve(0, 64)
    ids, pos = [3, 4, 5, 6], [0, 1, 2, 3]
    g = torch.Generator().manual_seed(0)
    hid = torch.randn(4, cfg.hidden, generator=g).to(torch.bfloat16)
    nxt = torch.tensor([4, 5, 6, 7], dtype=torch.int32)
    bg = BatchRows.make(ids, pos, [0] * 4, DEV, "all", 1, nsplit=2)
    bc = BatchRows.make(ids, pos, [0] * 4, "cpu", "all", 1)
    lg, hg = mg.mtp_forward(nxt.to(DEV), hid.to(DEV), bg, kvg)
    lc, hc = mc.mtp_forward(nxt, hid, bc, kvc)
    assert cos(lg.cpu(), lc) > 0.995 and cos(hg.cpu(), hc) > 0.999


def test_mtp_rounds_run_on_the_device_and_reproduce_plain_greedy():
    """Draft chain + verify step + acceptance count as one graph replay; the host reads one result vector per round."""
    from volta_engine_b200.runtime.engine import Engine
    from volta_engine_b200.runtime.mtp_runner import MtpRunner
    cfg = MLAConfig.tiny_mla(vocab=512)
    m = MLAModel(cfg, DEV).init_random(seed=1)
    prompt = torch.randint(0, cfg.vocab, (77,), generator=torch.Generator().manual_seed(4)).tolist()
    plain, _ = Engine(m, _kv(m, DEV), prefill_chunk=64).generate(prompt, 24)
    eng = Engine(m, _kv(m, DEV), prefill_chunk=64)
    run = MtpRunner(eng, depth=3)
    assert run._device_round_ok()
    eng.kv.reserve(0, len(prompt) + 40)
    tok = run.prefill_rows(0, prompt, 0, len(prompt), True)
    out, pos = [tok], len(prompt)
    while len(out) < 24:
        new = run.round(0, out[-1], pos)
        assert 1 <= len(new) <= 4
        out += new
        pos += len(new)
    assert out[:24] == plain[:24], (out, plain)
    assert run._sts[(1, 3)]["graph"] is not None and run.stats["rounds"] >= 6
    assert run.stats["proposed"] == 3 * run.stats["rounds"]
    # two slots in one joint round: one draft chain and one verify block of 8 rows; each slot continues its own greedy run
    other = torch.randint(0, cfg.vocab, (50,), generator=torch.Generator().manual_seed(9)).tolist()
    plain2, _ = Engine(m, _kv(m, DEV), prefill_chunk=64).generate(other, 16)
    eng2 = Engine(m, _kv(m, DEV), prefill_chunk=64)
    run2 = MtpRunner(eng2, depth=3)
    eng2.kv.reserve(0, len(prompt) + 40)
    eng2.kv.reserve(1, len(other) + 40)
    outs = [[run2.prefill_rows(0, prompt, 0, len(prompt), True)], [run2.prefill_rows(1, other, 0, len(other), True)]]
    poss = [len(prompt), len(other)]
    for _ in range(6):
        news = run2.round_joint([0, 1], [outs[0][-1], outs[1][-1]], poss)
        for j in range(2):
            outs[j] += news[j]
            poss[j] += len(news[j])
    n0, n1 = min(len(outs[0]), len(plain)), min(len(outs[1]), len(plain2))
    assert outs[0][:n0] == plain[:n0] and outs[1][:n1] == plain2[:n1] and n0 >= 7 and n1 >= 7, (outs, plain, plain2)
    assert run2._sts[(2, 3)]["graph"] is not None
    # the survival estimate shortens rounds whose later drafts are never accepted
    run2.adaptive = True
    run2.cond = [0.2, 0.2, 0.2]
    assert run2.round_depth() == 1
    run2.cond = [0.9, 0.9, 0.9]
    assert run2.round_depth() == 3
    from volta_engine_b200.ops import kernels as K
    assert K.check_status(DEV) == 0


@pytest.mark.parametrize("heads,nope,vd,shift", [(3, 128, 128, 0), (8, 96, 72, 1), (2, 256, 256, 0), (5, 37, 33, 3)])
@pytest.mark.parametrize("rows", [1, 3, 4, 5, 8, 9, 16, 17, 40])
def test_query_absorption_and_output_expansion(heads, nope, vd, shift, rows):
    """Every count of rows a launch is built for and more than one pass, widths that are no multiple of a piece, absorption weights that start
    between 16-byte boundaries. fp32 sums of exact products, rounded to bf16 once."""
    from volta_engine_b200._lib import call, ptr
    g = torch.Generator().manual_seed(rows)
    q = torch.randn(rows, heads * (nope + 64), generator=g).to(torch.bfloat16).to(DEV)
    wuk = torch.empty(heads * nope * 512 + 8, dtype=torch.bfloat16, device=DEV)[shift:shift + heads * nope * 512].view(heads, nope, 512)
    wuk.copy_(torch.randn(heads, nope, 512, generator=g))
    wuv = torch.randn(heads, vd, 512, generator=g).to(torch.bfloat16).to(DEV)
    q_abs = torch.full((rows, heads, 576), 7.0, dtype=torch.bfloat16, device=DEV)
    call("mla_absorb_q", "pliippii", ptr(q), q.stride(0), nope + 64, nope, ptr(wuk), ptr(q_abs), rows, heads)
    qh = q.view(rows, heads, nope + 64)
    want = torch.einsum("rhd,hdc->rhc", qh[..., :nope].double(), wuk.double())
    assert float((q_abs[..., :512].double() - want).norm() / want.norm()) < 2 ** -8
    assert torch.equal(q_abs[..., 512:], qh[..., nope:])
    o = torch.randn(rows, heads, 512, generator=g).to(torch.bfloat16).to(DEV)
    out = torch.full((rows, heads * vd), 7.0, dtype=torch.bfloat16, device=DEV)
    call("mla_expand_out", "pppliii", ptr(o), ptr(wuv), ptr(out), out.stride(0), rows, heads, vd)
    want = torch.einsum("rhc,hvc->rhv", o.double(), wuv.double()).reshape(rows, -1)
    assert float((out.double() - want).norm() / want.norm()) < 2 ** -8


@pytest.mark.parametrize("heads", [1, 7, 8, 20])
@pytest.mark.parametrize("rows", [5, 511, 512, 700])
@pytest.mark.parametrize("interleaved", [0, 1])
def test_latent_rotation_and_store_of_many_rows(heads, rows, interleaved):
    """Both forms of the launch, a block for eight heads of a row and a block for all of them; padding rows store nothing."""
    from volta_engine_b200._lib import call, ptr
    from volta_engine_b200.ops.reference import rope_rotate
    g = torch.Generator().manual_seed(rows + heads)
    q = torch.randn(rows, heads * 96, generator=g).to(torch.bfloat16)
    ckv, kr = torch.randn(rows, 512, generator=g).to(torch.bfloat16), torch.randn(rows, 64, generator=g).to(torch.bfloat16)
    pos = torch.arange(3, 3 + rows, dtype=torch.int32)
    slot = torch.ones(rows, dtype=torch.int32)
    slot[1] = -1
    table = torch.randperm(24, generator=g).int().reshape(2, 12)
    pool = torch.full((24, 1, 64, 576), 7.0, dtype=torch.bfloat16, device=DEV)
    a = [t.to(DEV) for t in (q, ckv, kr, pos, slot, table)]
    call("mla_rope_store", "pliiplplpppipifi", ptr(a[0]), a[0].stride(0), 96, heads, ptr(a[1]), 512, ptr(a[2]), 64, ptr(a[3]), ptr(a[4]),
         ptr(a[5]), 12, ptr(pool), rows, 10000.0, interleaved)
    want = q.view(rows, heads, 96).clone()
    want[..., 32:] = rope_rotate(want[..., 32:].contiguous(), pos, 64, 10000.0, bool(interleaved))
    got = a[0].cpu().view(rows, heads, 96)
    assert torch.equal(got[..., :32], q.view(rows, heads, 96)[..., :32])
    assert float((got.float() - want.float()).abs().max()) < 3e-2                 # (an ulp of bf16 at 4)
    lat = torch.cat([ckv, rope_rotate(kr.view(rows, 1, 64).clone(), pos, 64, 10000.0, bool(interleaved))[:, 0]], 1)
    want_pool = torch.full((24, 64, 576), 7.0)
    for r in range(rows):
        if slot[r] >= 0:
            want_pool[table[1, pos[r] // 64], pos[r] % 64] = lat[r].float()
    assert float((pool.cpu()[:, 0].float() - want_pool).abs().max()) < 3e-2
