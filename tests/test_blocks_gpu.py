"""Block-quantised mat-vecs and grouped GEMMs at the edges of their tiles, against the block decoders of quant/gguf.py and quant/exl3.py."""
import pytest
import torch

from volta_engine_b200.ops.linear_gguf import FUSED_TYPES, LinearGGUF
from volta_engine_b200.quant import gguf as gq

pytestmark = pytest.mark.gpu
TYPES = sorted(FUSED_TYPES)


def _rel(a, b):
    return float((a.double() - b.double()).norm() / (b.double().norm() + 1e-30))


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("shift", [0, 1, 2, 6])
def test_gguf_matvec_edges(t, shift):
    """Rows around tiles of 16 and 32, K of one chunk to more units than warps with partial last units, every count of activation rows, and
    blocks that start at odd and at 2-byte addresses (``shift`` bytes into their allocation). fp32 sums of at most 4608 products: 1e-5;
    a row's result does not depend on the rows beside it."""
    big = gq.BLOCK[t][0] == 256
    for N, K in ((1, 256), (17, 512), (33, 2304), (100, 4608)) if big else ((1, 32), (17, 96), (33, 1056), (100, 4448)):
        raw = gq.random_blocks(t, N, K, seed=t + N, amp=0.05)
        w = gq.dequantize(raw, t, K).double()
        buf = torch.zeros(raw.numel() + 64, dtype=torch.uint8, device="cuda")
        view = buf[shift:shift + raw.numel()].view(N, -1)
        view.copy_(raw.reshape(N, -1))
        lin = LinearGGUF(view, t, N, K)
        assert lin.raw.data_ptr() == view.data_ptr()
        x = torch.randn(16, K, generator=torch.Generator().manual_seed(N)).to(torch.bfloat16)
        full = lin.forward(x.cuda(), out_f32=True)
        want = x.double() @ w.t()
        assert _rel(full.cpu(), want) < 1e-5, (t, N, K)
        for M in (1, 4, 5, 8, 9):
            assert torch.equal(lin.forward(x[:M].cuda(), out_f32=True), full[:M]), (t, N, K, M)
        assert _rel(lin.forward(x[:3].cuda()).cpu(), want[:3]) < 2 ** -8      # bf16 output: half a unit in the last place


@pytest.mark.parametrize("t", TYPES)
def test_gguf_matvec_in_lane_order(t):
    """Asked for it, the mat-vec gives bit for bit what the byte-by-byte kernel gives, which the same blocks at an odd address take: every
    count of rows a launch is built for, K of less than one step of 1024 weights to several with a partial last one."""
    big = gq.BLOCK[t][0] == 256
    for N, K in ((1, 256), (17, 1024), (35, 2304), (16, 4608)) if big else ((1, 32), (17, 1024), (35, 1056), (16, 4448)):
        raw = gq.random_blocks(t, N, K, seed=t + K, amp=0.05)
        x = torch.randn(16, K, generator=torch.Generator().manual_seed(N)).to(torch.bfloat16).cuda()
        lins = []
        for shift in (1, 0, 2, 6):
            buf = torch.zeros(raw.numel() + 64, dtype=torch.uint8, device="cuda")
            view = buf[shift:shift + raw.numel()].view(N, -1)
            view.copy_(raw.reshape(N, -1))
            lins.append(LinearGGUF(view, t, N, K, ordered=True))
        for M in (1, 2, 4, 5, 8, 9, 16):
            want = lins[0].forward(x[:M], out_f32=True)
            for lin in lins[1:]:
                assert torch.equal(lin.forward(x[:M], out_f32=True), want), (t, N, K, M)
            assert torch.equal(lins[1].forward(x[:M]), lins[0].forward(x[:M]))


@pytest.mark.parametrize("spec", ["gguf_iq1_m", "gguf_q8_0+q4_k", "gguf_q2_k+q6_k", "gguf_iq3_s+iq4_xs", "gguf_q5_0+q4_1", "gguf_iq2_xxs+iq4_nl"])
def test_gguf_experts_in_lane_order(spec):
    """The same for routed mat-vecs, with both activations and a limit; experts elsewhere give zeros."""
    from volta_engine_b200.ops.moe_gguf import GGUFExpertBank, parse_expert_quant
    gt, dt = parse_expert_quant(spec)
    E, I, H = 4, 256, 1536
    bank = GGUFExpertBank.random(E, I, H, gt, dt, e0=1, seed=5, amp=0.05, device="cuda")

    def odd(raw):
        buf = torch.zeros(raw.numel() + 16, dtype=torch.uint8, device="cuda")
        buf[1:1 + raw.numel()] = raw.reshape(-1)
        return buf[1:1 + raw.numel()].reshape(raw.shape)
    other = GGUFExpertBank(odd(bank.gu_raw), gt, odd(bank.dn_raw), dt, 1, I, H)
    g = torch.Generator().manual_seed(9)
    x = torch.randn(7, H, generator=g).to(torch.bfloat16).cuda()
    ids = torch.stack([torch.randperm(6, generator=g)[:3] for _ in range(7)]).to(torch.int32).cuda()
    for act, limit in ((0, 0.0), (1, 0.0), (0, 0.5)):
        got = bank.routes(x, ids, act, limit, ordered=True)
        assert torch.equal(got, other.routes(x, ids, act, limit)) and got.any()
    assert not got[((ids < 1) | (ids >= 5)).reshape(-1)].any()


@pytest.mark.parametrize("t", TYPES)
def test_gguf_matvec_is_as_near_as_sums_weight_by_weight(t):
    """Distance to 64 bits over a long K against that of the same blocks at an odd address, which are summed weight by weight in fp32."""
    N, K, far = 64, 17408, []
    raw = gq.random_blocks(t, N, K, seed=t, amp=0.05)
    w = gq.dequantize(raw, t, K).double().cuda()
    x = torch.randn(16, K, generator=torch.Generator().manual_seed(t)).to(torch.bfloat16).cuda()
    for shift in (0, 1):
        buf = torch.zeros(raw.numel() + 64, dtype=torch.uint8, device="cuda")
        view = buf[shift:shift + raw.numel()].view(N, -1)
        view.copy_(raw.reshape(N, -1))
        far.append(_rel(LinearGGUF(view, t, N, K).forward(x, out_f32=True), x.double() @ w.t()))
    assert far[0] < 1.1 * far[1], (t, far)


def _non_finite(K):
    """Four rows of activations: none, an infinity, an infinity of each sign in different chunks, values whose products with a block's
    integers overflow where those with its weights do not."""
    x = torch.randn(4, K, generator=torch.Generator().manual_seed(K)).to(torch.bfloat16)
    x[1, 37] = float("inf")
    x[2, 5], x[2, K - 3] = float("inf"), float("-inf")
    x[3, ::2] = 3e37
    return x.cuda()


def _same_where_not_finite(got, want, bound):
    """Infinities and NaN in the same places with the same signs; numbers within 1e-5 of the sum of the products' magnitudes."""
    fine = torch.isfinite(want)
    assert torch.equal(got[~fine].nan_to_num(7.0), want[~fine].nan_to_num(7.0))
    assert bool((((got - want).double().abs() <= 1e-5 * bound)[fine]).all())


@pytest.mark.parametrize("t", TYPES)
def test_gguf_matvec_of_infinite_and_huge_activations(t):
    """Blocks at even addresses against blocks at an odd one, which are summed weight by weight."""
    N, K = 40, 512
    raw = gq.random_blocks(t, N, K, seed=t, amp=0.01)
    buf = torch.zeros(raw.numel() + 64, dtype=torch.uint8, device="cuda")
    odd = buf[1:1 + raw.numel()].view(N, -1)
    odd.copy_(raw.reshape(N, -1))
    x = _non_finite(K)
    got, want = (LinearGGUF(r, t, N, K).forward(x, out_f32=True) for r in (raw.cuda(), odd))
    w = gq.dequantize(raw, t, K).double().cuda()
    _same_where_not_finite(got, want, x.double().nan_to_num(0.0, 0.0, 0.0).abs() @ w.abs().t())
    assert torch.isinf(want[1]).any()


@pytest.mark.parametrize("spec", ["gguf_q4_k+q2_k", "gguf_q5_1+q4_1", "gguf_q5_k+q6_k", "gguf_iq1_m+iq2_s"])
def test_gguf_experts_of_infinite_and_huge_activations(spec):
    """The routed mat-vecs, the gated pair among them; outputs are bf16."""
    from volta_engine_b200.ops.moe_gguf import GGUFExpertBank, parse_expert_quant
    gt, dt = parse_expert_quant(spec)
    E, I, H = 3, 256, 512
    bank = GGUFExpertBank.random(E, I, H, gt, dt, seed=5, amp=0.01, device="cuda")

    def odd(raw):
        buf = torch.zeros(raw.numel() + 16, dtype=torch.uint8, device="cuda")
        buf[1:1 + raw.numel()] = raw.reshape(-1)
        return buf[1:1 + raw.numel()].reshape(raw.shape)
    other = GGUFExpertBank(odd(bank.gu_raw), gt, odd(bank.dn_raw), dt, 0, I, H)
    ids = torch.tensor([[0, 2], [1, 0], [2, 5], [0, 1]], dtype=torch.int32, device="cuda")
    x = _non_finite(H)
    got, want = bank.routes_decode(x, ids, 0, 0.0).float(), other.routes_decode(x, ids, 0, 0.0).float()
    fine = torch.isfinite(want)
    assert torch.equal(got[~fine].nan_to_num(7.0), want[~fine].nan_to_num(7.0)) and not fine.all()
    assert bool(((got - want).abs() <= 2 ** -6 * want.abs().amax(-1, keepdim=True))[fine].all())


@pytest.mark.parametrize("spec", ["gguf_q8_0+q4_0", "gguf_q4_k+q5_1", "gguf_iq1_m+iq2_xs", "gguf_q6_k+q3_k", "gguf_q2_k+iq4_xs"])
@pytest.mark.parametrize("rows", [17, 130, 700])
def test_gguf_experts_decoded_in_tiles(spec, rows):
    """The grouped GEMM that decodes blocks in its tile loader against decoding the bank to bf16 first: the same operands, sums of the same
    MMA. Experts with no row, one row and several tiles; feature counts that are no multiple of 128; a share of experts elsewhere."""
    from volta_engine_b200.ops.moe_gguf import GGUFExpertBank, parse_expert_quant
    gt, dt = parse_expert_quant(spec)
    E, I, H, k = 6, 256 + 64 * (gq.BLOCK[dt][0] == 32), 512, 3
    bank = GGUFExpertBank.random(E, I, H, gt, dt, e0=2, seed=rows, amp=0.05, device="cuda")
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, H, generator=g).to(torch.bfloat16).cuda()
    ids = torch.stack([torch.randperm(9, generator=g)[:k] for _ in range(rows)]).to(torch.int32)
    ids[:, 0] = 5
    ids[ids == 4] = 8
    ids[0, 1] = 4                                   # expert 4: one row; 0, 1 and 8: elsewhere
    ids = ids.cuda()
    assert bank._decodes_in_tiles(rows * k)
    got, want = bank.routes_prefill(x, ids, 0, 0.0), bank._routes_prefill_slabs(x, ids, 0, 0.0)
    away = ((ids < 2) | (ids >= 8)).reshape(-1)
    assert not got[away].any()
    assert _rel(got, want) < 1e-3
    from volta_engine_b200.ops import kernels as K
    assert K.check_status("cuda") == 0


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("I,rows", [(256, 33), (512, 150)])
def test_gguf_experts_of_every_format_decoded_in_tiles(t, I, rows):
    """Bit for bit the bank decoded to bf16 first: the same operands in the same chain over K. (Formats of 32-weight blocks also with a K that
    ends inside a staged unit.)"""
    from volta_engine_b200.ops.moe_gguf import GGUFExpertBank
    big = gq.BLOCK[t][0] == 256
    E, H, k = 3, 512, 2
    I += 0 if big else 32
    bank = GGUFExpertBank.random(E, I, H, t, t, seed=t, amp=0.05, device="cuda")
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, H, generator=g).to(torch.bfloat16).cuda()
    ids = torch.stack([torch.randperm(4, generator=g)[:k] for _ in range(rows)]).to(torch.int32).cuda()
    assert bank._decodes_in_tiles(rows * k)
    assert torch.equal(bank.routes_prefill(x, ids, 0, 0.0), bank._routes_prefill_slabs(x, ids, 0, 0.0))
    from volta_engine_b200.ops import kernels as K
    assert K.check_status("cuda") == 0


@pytest.mark.parametrize("spec,gu_at,dn_at", [("gguf_q4_k+q6_k", 2, 0), ("gguf_q6_k+q4_k", 2, 2), ("gguf_iq1_s+q4_1", 4, 2), ("gguf_q8_0+q8_0", 2, 6)])
def test_gguf_experts_at_any_even_address(spec, gu_at, dn_at):
    """A bank inside a larger allocation gives what it gives at the start of one, whichever way its formats and addresses let it take."""
    from volta_engine_b200.ops.moe_gguf import GGUFExpertBank, parse_expert_quant
    gt, dt = parse_expert_quant(spec)
    E, I, H, k, rows = 3, 256, 512, 2, 50
    bank = GGUFExpertBank.random(E, I, H, gt, dt, seed=5, amp=0.05, device="cuda")

    def at(raw, off):
        buf = torch.zeros(raw.numel() + 16, dtype=torch.uint8, device="cuda")
        buf[off:off + raw.numel()] = raw.reshape(-1)
        return buf[off:off + raw.numel()].reshape(raw.shape)
    moved = GGUFExpertBank(at(bank.gu_raw, gu_at), gt, at(bank.dn_raw, dn_at), dt, 0, I, H)
    assert moved.gu_raw.data_ptr() % 16 == gu_at and moved.dn_raw.data_ptr() % 16 == dn_at
    g = torch.Generator().manual_seed(3)
    x = torch.randn(rows, H, generator=g).to(torch.bfloat16).cuda()
    ids = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(rows)]).to(torch.int32).cuda()
    assert _rel(moved.routes_prefill(x, ids, 0, 0.0), bank._routes_prefill_slabs(x, ids, 0, 0.0)) < 1e-3


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("cb", [0, 1, 2])
def test_exl3_experts_decoded_in_tiles(bits, cb):
    """The same for trellis codes; K of the down projection is no multiple of the 256 weights a unit holds."""
    from volta_engine_b200.ops.moe_exl3 import EXL3ExpertBank
    E, I, H, k, rows = 4, 128, 384, 2, 150
    bank = EXL3ExpertBank.random(E, I, H, bits, e0=1, seed=bits, device="cuda", std=0.05)
    bank.cb = cb
    g = torch.Generator().manual_seed(bits)
    x = torch.randn(rows, H, generator=g).to(torch.bfloat16).cuda()
    ids = torch.stack([torch.randperm(6, generator=g)[:k] for _ in range(rows)]).to(torch.int32).cuda()
    got, want = bank.routes_prefill(x, ids, 0, 0.0), bank._routes_prefill_slabs(x, ids, 0)
    away = ((ids < 1) | (ids >= 5)).reshape(-1)
    assert not got[away].any() and not want[away].any()
    assert _rel(got, want) < 1e-3
    few = bank.routes_decode(x[:5], ids[:5], 0, 0.0)
    assert not few[away[:5 * k]].any()
    assert _rel(few, want[:5 * k]) < 2e-2           # fp16 activations against bf16 ones
    from volta_engine_b200.ops import kernels as K
    assert K.check_status("cuda") == 0


@pytest.mark.parametrize("rows", [1, 5, 40])
def test_exl3_experts_take_ids_of_any_integer_type_and_stride(rows):
    """Decode rows and a prompt: 64-bit, 16-bit and strided ids name the same experts as dense 32-bit ones."""
    from volta_engine_b200.ops.moe_exl3 import EXL3ExpertBank
    E, I, H, k = 4, 128, 256, 2
    bank = EXL3ExpertBank.random(E, I, H, 4, e0=1, seed=7, device="cuda", std=0.05)
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, H, generator=g).to(torch.bfloat16).cuda()
    ids = torch.stack([torch.randperm(6, generator=g)[:k] for _ in range(rows)]).to(torch.int32).cuda()
    want = bank.routes(x, ids, 0, 0.0)
    wide = torch.full((rows, 3 * k), 3, dtype=torch.int32, device="cuda")
    wide[:, ::3] = ids
    for form in (ids.long(), ids.short(), wide[:, ::3], ids.t().contiguous().t(), ids.long().t().contiguous().t()):
        assert torch.equal(bank.routes(x, form, 0, 0.0), want), (form.dtype, form.stride())
    assert want.any()


@pytest.mark.parametrize("N,K", [(1, 8), (17, 40), (512, 7168), (2368, 264), (2369, 1032), (5000, 2048)])
def test_bf16_matvec_edges(N, K):
    """Row counts on both sides of the warp-count rule, K that ends inside a 32-wide step, every count of activation rows up to more than
    one pass; fp32 sums of exact products (1e-5), a row's result independent of the rows beside it."""
    from volta_engine_b200.ops import kernels as K_
    g = torch.Generator().manual_seed(N)
    W, x = torch.randn(N, K, generator=g).to(torch.bfloat16), torch.randn(21, K, generator=g).to(torch.bfloat16)
    full = K_.bf16_gemv_f32(W.cuda(), x.cuda())
    assert _rel(full.cpu(), x.double() @ W.double().t()) < 1e-5
    for M in (1, 2, 3, 7, 8, 9, 16):
        assert torch.equal(K_.bf16_gemv_f32(W.cuda(), x[:M].cuda()), full[:M]), M


@pytest.mark.parametrize("bits", [1, 3, 4, 6, 8])
def test_exl3_matvec_units_and_groups(bits):
    """More and fewer units than resident blocks, units of fewer than four column tiles, K of fewer k-tiles than warps, groups without an
    expert between others, codes that start on a 4-byte boundary; against the product with the matrix decoded to bf16 (2^-8)."""
    from volta_engine_b200.ops.linear_exl3 import exl3_gemv, exl3_reconstruct
    g = torch.Generator().manual_seed(bits)
    for E, K, N, groups, M in ((1, 16, 16, 1, 16), (3, 80, 48, 7, 1), (2, 1040, 176, 300, 2), (2, 256, 64, 5, 9), (2, 272, 112, 200, 1)):
        n = (K // 16) * (N // 16) * 16 * bits
        raw = torch.randint(-32768, 32768, (E * n + 8,), generator=g, dtype=torch.int32).to(torch.int16).cuda()
        x = torch.randn(groups * M, K, generator=g).half().cuda()
        e = torch.randint(-1, E, (groups,), generator=g, dtype=torch.int32).cuda()
        e[0] = 0
        for shift in (0, 2):
            codes = raw[shift:shift + E * n]
            y = exl3_gemv(codes, x, M, K, N, bits, 2, out=torch.full((groups * M, N), 7.0, device="cuda"), expert=e, expert_stride=n, groups=groups)
            for gi in range(0, groups, 1 if groups < 20 else 23):
                got = y[gi * M:(gi + 1) * M]
                if int(e[gi]) < 0:
                    assert bool((got == 7.0).all())
                    continue
                w = exl3_reconstruct(codes[int(e[gi]) * n:(int(e[gi]) + 1) * n].clone(), K, N, bits, 2)
                want = x[gi * M:(gi + 1) * M].double() @ w.double().t()
                assert _rel(got, want) < 2 ** -8, (bits, K, N, gi)


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two devices")
def test_kernels_of_much_shared_memory_run_on_every_device():
    """What a kernel is allowed belongs to a device: one process may use a second one after the first."""
    from volta_engine_b200._lib import call, ptr
    from volta_engine_b200.ops.linear_exl3 import exl3_gemv
    out = []
    for dev in (0, 1, 0):
        with torch.cuda.device(dev):
            g = torch.Generator().manual_seed(1)
            x = torch.randn(9, 512, generator=g).to(torch.bfloat16).cuda()
            raw = gq.random_blocks(12, 64, 512, seed=1, amp=0.05).cuda()
            ys = [LinearGGUF(raw, 12, 64, 512, ordered=o).forward(x) for o in (False, True)]
            codes = torch.randint(-32768, 32768, (32 * 8 * 64,), generator=g, dtype=torch.int32).to(torch.int16).cuda()
            e = torch.zeros(60, dtype=torch.int32, device="cuda")
            ys.append(exl3_gemv(codes, torch.randn(60, 512, generator=g).half().cuda(), 1, 512, 128, 4, 2, expert=e, expert_stride=codes.numel(), groups=60))
            o, w = torch.randn(3, 2, 512, generator=g).to(torch.bfloat16).cuda(), torch.randn(2, 64, 512, generator=g).to(torch.bfloat16).cuda()
            y = torch.empty(3, 128, dtype=torch.bfloat16, device="cuda")
            call("mla_expand_out", "pppliii", ptr(o), ptr(w), ptr(y), y.stride(0), 3, 2, 64)
            out.append([t.cpu() for t in ys + [y]])
    for other in out[1:]:
        assert all(torch.equal(a, b) for a, b in zip(out[0], other))
