"""Tensor-core prefill: rows at the edges of a warp (32), of a Q tile (128) and of an item (256), heads and batches that lie
next to one another in either row order, items that follow one another in a CTA, and a running maximum that moves late."""
import pytest
import torch

from tests import helpers

pytestmark = pytest.mark.gpu


def _float64(q, k, v, scale, causal, prefix):
    group = q.shape[1] // k.shape[1]
    kk, vv = (t.double().repeat_interleave(group, 1) for t in (k, v))
    scores = q.double() @ kk.transpose(-1, -2) * scale
    if causal:
        visible = torch.ones(scores.shape[-2:], dtype=torch.bool, device="cuda").tril(prefix)
        scores = scores.masked_fill(~visible, float("-inf"))
    return torch.softmax(scores, -1) @ vv, torch.logsumexp(scores, -1)


# batch, q_heads, kv_heads, rows, prefix, causal; the last two have more items than SMs
@pytest.mark.parametrize("shape", [(2, 3, 3, 1, 0, True), (2, 3, 1, 31, 5, True), (1, 4, 2, 33, 0, False), (2, 2, 2, 127, 130, True),
                                   (1, 2, 2, 129, 0, True), (2, 2, 1, 257, 0, True), (1, 2, 2, 385, 100, False), (3, 40, 8, 400, 0, True),
                                   (2, 64, 64, 300, 61, True)])
@pytest.mark.parametrize("token_major", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_row_edges_match_float64(backend, shape, token_major, dtype):
    b, hq, hkv, rows, prefix, causal = shape
    gen = torch.Generator(device="cuda").manual_seed(rows + prefix)
    q, k, v = (torch.randn(b, h, n, 128, device="cuda", generator=gen).to(dtype) for h, n in ((hq, rows), (hkv, prefix + rows), (hkv, prefix + rows)))
    k[:, :, -40:] *= 6   # the row maxima move by more than the carried reference allows in the last tiles
    lse = torch.empty(b, hq, rows, device="cuda")
    # The output lies inside a larger buffer: nothing in front of its first row or behind its last one may change.
    guard, size = 4096, b * hq * rows * 128
    buffer = torch.full((size + 2 * guard,), float("nan"), device="cuda", dtype=dtype)
    buffer[:guard] = buffer[-guard:] = 7.0
    out = buffer[guard:-guard].view((b, rows, hq, 128) if token_major else (b, hq, rows, 128))
    for values in (-v, v):   # back to back: the second launch overwrites what the first one writes
        backend.attention_fa(q, k, values, 128 ** -0.5, causal, out=out, lse=lse, query_start=prefix, token_major_out=token_major)
    torch.cuda.synchronize()
    backend.poll()
    assert (buffer[:guard] == 7.0).all() and (buffer[-guard:] == 7.0).all()
    if token_major:
        out = out.transpose(1, 2)
    want, want_lse = _float64(q, k, v, 128 ** -0.5, causal, prefix)
    # 16-bit storage: P and the result are rounded once each, by 2^-9 at most, so a row's 128 values are off by about 2^-9 of their
    # norm; also where the row is small beside others
    assert helpers.max_rel_err(out.double().cpu().numpy(), want.cpu().numpy()) <= 1e-2
    assert ((out.double() - want).norm(dim=-1) / want.norm(dim=-1)).max().item() <= 1e-2
    assert (lse.double() - want_lse).abs().max().item() <= 1e-3
