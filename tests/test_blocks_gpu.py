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
