"""f32 prefill through the register-tiled kernel: tile edges of rows (32) and keys (64, two groups), masks, grouped heads and
token-major rows against float64; keys a row does not see must not reach its arithmetic."""
import pytest
import torch

from tests import helpers

pytestmark = pytest.mark.gpu


# batch, q_heads, kv_heads, rows, prefix, head_dim, causal
@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 0, 64, False), (1, 2, 1, 31, 0, 64, True), (2, 2, 2, 33, 32, 128, True), (1, 4, 2, 64, 64, 128, False),
                                   (1, 2, 2, 65, 127, 64, True), (1, 3, 3, 129, 0, 128, True), (1, 2, 1, 200, 313, 64, False)])
@pytest.mark.parametrize("token_major", [False, True])
def test_tile_edges_match_float64(backend, shape, token_major):
    b, hq, hkv, rows, prefix, d, causal = shape
    keys = prefix + rows
    gen = torch.Generator(device="cuda").manual_seed(rows + keys)
    q, k, v = (torch.randn(b, h, n, d, device="cuda", generator=gen) for h, n in ((hq, rows), (hkv, keys), (hkv, keys)))
    visible = torch.ones(rows, keys, dtype=torch.bool, device="cuda")
    if causal:
        visible = visible.tril(prefix)
        v[:, :, -1] = float("inf")   # only the last row sees this key
    lse, m, l = (torch.empty(b, hq, rows, device="cuda") for _ in range(3))
    out = backend.attention_fa(q, k, v, d ** -0.5, causal, lse=lse, row_max=m, row_sum=l, query_start=prefix, token_major_out=token_major)
    torch.cuda.synchronize()
    backend.poll()
    if token_major:
        out = out.transpose(1, 2)
    kk, vv = (t.double().repeat_interleave(hq // hkv, 1) for t in (k, v))
    scores = (q.double() @ kk.transpose(-1, -2) * d ** -0.5).masked_fill(~visible, float("-inf"))
    finite = rows - 1 if causal else rows
    if causal:
        assert torch.isinf(out[:, :, -1]).all()
        vv[:, :, -1] = 0
    want = (torch.softmax(scores, -1) @ vv)[:, :, :finite]
    if finite:
        assert helpers.max_rel_err(out[:, :, :finite].double().cpu().numpy(), want.cpu().numpy()) <= 1e-5   # the f32 bound of the path
    assert (lse.double() - torch.logsumexp(scores, -1)).abs().max().item() <= 1e-5
    assert (m.double() - scores.amax(-1)).abs().max().item() <= 1e-5
    assert torch.allclose(m.double() + l.double().log(), lse.double(), atol=1e-5)


@pytest.mark.parametrize("keys", [1, 64, 65, 128, 192, 193, 256, 257, 320, 513])
@pytest.mark.parametrize("causal", [False, True])
def test_key_tiles_over_the_groups_match_float64(backend, keys, causal):
    # 64-key tiles go to four groups of threads in turn: none, some or all of them with a tile, whole, ragged or on the diagonal
    rows, d = min(keys, 70), 64
    gen = torch.Generator(device="cuda").manual_seed(keys)
    q, k, v = (torch.randn(2, 3, n, d, device="cuda", generator=gen) for n in (rows, keys, keys))
    lse = torch.empty(2, 3, rows, device="cuda")
    out = backend.attention_fa(q, k, v, d ** -0.5, causal, lse=lse, query_start=keys - rows)
    torch.cuda.synchronize()
    backend.poll()
    scores = q.double() @ k.double().transpose(-1, -2) * d ** -0.5
    if causal:
        scores = scores.masked_fill(~torch.ones(rows, keys, dtype=torch.bool, device="cuda").tril(keys - rows), float("-inf"))
    want = torch.softmax(scores, -1) @ v.double()
    assert helpers.max_rel_err(out.double().cpu().numpy(), want.cpu().numpy()) <= 1e-5   # the f32 bound of the path
    assert (lse.double() - torch.logsumexp(scores, -1)).abs().max().item() <= 1e-5


@pytest.mark.parametrize("batch,heads,rows,keys", [(1, 37, 128, 129), (1, 37, 129, 129), (5, 4, 256, 257), (3, 7, 256, 257), (2, 75, 33, 500), (2, 37, 33, 65)])
@pytest.mark.parametrize("causal", [False, True])
def test_either_number_of_groups_matches_float64(backend, batch, heads, rows, keys, causal):
    # launches on both sides of the lines between two and four groups: 148 blocks of 32 rows, 20 causal heads, 128 keys
    gen = torch.Generator(device="cuda").manual_seed(heads + keys)
    q, k, v = (torch.randn(batch, heads, n, 64, device="cuda", generator=gen) for n in (rows, keys, keys))
    lse = torch.empty(batch, heads, rows, device="cuda")
    out = backend.attention_fa(q, k, v, 64 ** -0.5, causal, lse=lse, query_start=keys - rows)
    torch.cuda.synchronize()
    backend.poll()
    scores = q.double() @ k.double().transpose(-1, -2) * 64 ** -0.5
    if causal:
        scores = scores.masked_fill(~torch.ones(rows, keys, dtype=torch.bool, device="cuda").tril(keys - rows), float("-inf"))
    want = torch.softmax(scores, -1) @ v.double()
    assert helpers.max_rel_err(out.double().cpu().numpy(), want.cpu().numpy()) <= 1e-5   # the f32 bound of the path
    assert (lse.double() - torch.logsumexp(scores, -1)).abs().max().item() <= 1e-5
