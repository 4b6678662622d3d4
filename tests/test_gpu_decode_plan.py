"""Decode with the library's own plan (kv_splits = 0): one cluster per (batch, KV head) for short caches, several with a fold
of records for long ones, narrow (up to 8 query heads per KV head) and wide groups, caches shorter than a warp's tile."""
import pytest
import torch

from tests import helpers

pytestmark = pytest.mark.gpu


# batch, q_heads, kv_heads, capacity, visible keys
@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 1), (1, 4, 4, 64, 63), (1, 7, 1, 65, 65), (2, 8, 1, 513, 512), (1, 9, 1, 520, 513),
                                   (1, 16, 1, 2100, 2049), (1, 2, 2, 20000, 19999), (3, 28, 4, 700, 700), (40, 32, 8, 130, 129)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_decode_plans_match_float64(backend, shape, dtype):
    b, hq, hkv, capacity, visible = shape
    gen = torch.Generator(device="cuda").manual_seed(capacity + visible)
    q, k, v = (torch.randn(b, h, n, 128, device="cuda", generator=gen).to(dtype) for h, n in ((hq, 1), (hkv, capacity), (hkv, capacity)))
    k[:, :, visible:] = float("nan")   # keys behind the cache's end must not be touched by the arithmetic
    v[:, :, visible:] = float("nan")
    lse, m, l = (torch.empty(b, hq, 1, device="cuda") for _ in range(3))
    for _ in range(2):   # the arrival counters are left ready for the next call
        out = backend.attention_fd(q, k, v, 128 ** -0.5, lse=lse, row_max=m, row_sum=l, key_end=visible)
    torch.cuda.synchronize()
    backend.poll()
    kk, vv = (t[:, :, :visible].double().repeat_interleave(hq // hkv, 1) for t in (k, v))
    scores = q.double() @ kk.transpose(-1, -2) * 128 ** -0.5
    want = torch.softmax(scores, -1) @ vv
    # P and the result are each rounded once to the storage type: 2 x 2^-9 (bf16), 2 x 2^-12 (f16) of the largest value, doubled
    bound = 2 ** -7 if dtype == torch.bfloat16 else 2 ** -10
    assert helpers.max_rel_err(out.double().cpu().numpy(), want.cpu().numpy()) <= bound
    assert (lse.double() - torch.logsumexp(scores, -1)).abs().max().item() <= 2e-4
    assert (m.double() - scores.amax(-1)).abs().max().item() <= 1e-4
    assert torch.allclose(m.double() + l.double().log(), lse.double(), atol=1e-5)


@pytest.mark.parametrize("static", [False, True])
def test_decode_is_right_after_calls_that_overlapped(backend, static):
    """Calls that share the scratch and overlap on two streams have no defined result, but the calls after them do, eager and
    replayed from a graph, with every number of records."""
    gen = torch.Generator(device="cuda").manual_seed(17)
    q, k, v = (torch.randn(2, h, n, 128, device="cuda", generator=gen).bfloat16() for h, n in ((8, 1), (2, 30000), (2, 30000)))
    kk, vv = (t.double().repeat_interleave(4, 1) for t in (k, v))
    want = torch.softmax(q.double() @ kk.transpose(-1, -2) * 128 ** -0.5, -1) @ vv
    decode = backend.attention_fd_static if static else backend.attention_fd

    def run(splits, **more):
        return decode(q, k, v, 128 ** -0.5, kv_splits=splits, **more)
    run(16)   # the scratch has its size
    torch.cuda.synchronize()
    graph, replayed = torch.cuda.CUDAGraph(), torch.empty_like(q)
    with torch.cuda.graph(graph):
        run(6, out=replayed)
    streams = [torch.cuda.Stream() for _ in range(2)]
    spare = [torch.empty_like(q) for _ in streams]
    for turn in range(4):
        for _ in range(8):
            for stream, splits, out in zip(streams, (3 + turn, 7), spare):
                run(splits, stream=stream.cuda_stream, out=out)
        torch.cuda.synchronize()
        for splits in (2, 7, 16):
            got = run(splits, out=torch.full_like(q, float("nan")))
            assert helpers.max_rel_err(got.double().cpu().numpy(), want.cpu().numpy()) <= 2 ** -7
        replayed.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert helpers.max_rel_err(replayed.double().cpu().numpy(), want.cpu().numpy()) <= 2 ** -7
    backend.poll()
