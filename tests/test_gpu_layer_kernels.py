"""Kernels of the decoder layer at the widths and sizes where their branches meet."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [4, 20, 64, 128, 1040, 1028])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_rope_split_widths(backend, hd, dtype):
    # both access widths (head_dim a multiple of 16 or not) and more angles than fit in shared memory at a time
    batch, seq, hq, hkv, offset = 2, 9, 3, 1, 777
    g = torch.Generator(device="cpu").manual_seed(hd)
    qkv = torch.randn(batch * seq, (hq + 2 * hkv) * hd, generator=g).to(dtype)
    q, k, v = (t.cpu() for t in backend.rope_split(qkv.cuda(), batch, seq, hq, hkv, hd, 10000.0, position_offset=offset))
    rows = qkv.reshape(batch, seq, hq + 2 * hkv, hd).permute(0, 2, 1, 3)
    assert torch.equal(v, rows[:, hq + hkv:])
    angle = (offset + torch.arange(seq).double())[:, None] * 10000.0 ** (-torch.arange(0, hd, 2).double() / hd)
    x = rows[:, :hq + hkv].double()
    lo, hi = x[..., : hd // 2], x[..., hd // 2:]
    want = torch.cat((lo * angle.cos() - hi * angle.sin(), hi * angle.cos() + lo * angle.sin()), -1)
    # the f32 angle of up to 786 radians is off by about 786 * 2^-22; then one rounding to 8 (bf16) or 11 (f16) significant
    # bits, which is off by at most 2^-8 or 2^-11 of the value
    bound = want.abs().max().item() * ((2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) + 786 * 2.0 ** -22)
    assert (torch.cat((q, k), 1).double() - want).abs().max().item() <= bound
