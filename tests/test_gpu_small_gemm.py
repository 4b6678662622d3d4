"""GEMM regions of few rows or few columns (one 64- or 128-column tile per CTA, 16 to 256 rows): tile edges, remainders of K,
every orientation and epilogue against float64, and the rows' bits against the same rows inside a large problem."""
import pytest
import torch

from tests import helpers
from vibe_compiler_b200 import _abi as abi

pytestmark = pytest.mark.gpu


def operands(m, n, k, dtype, lt, rt):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.rand((k, m) if lt else (m, k), device="cuda", generator=gen).mul_(2).sub_(1).to(dtype)
    b = torch.rand((n, k) if rt else (k, n), device="cuda", generator=gen).mul_(2).sub_(1).to(dtype)
    return a, b


@pytest.mark.parametrize("m,n,k", [(8, 8, 8), (8, 64, 64), (16, 72, 136), (24, 136, 1032), (64, 512, 128), (72, 8, 200), (104, 4096, 192),
                                   (136, 256, 264), (256, 128, 2048), (264, 1024, 72), (8, 20000, 256)])
@pytest.mark.parametrize("lt,rt", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_tile_edges_match_float64(backend, m, n, k, lt, rt, dtype):
    a, b = operands(m, n, k, dtype, lt, rt)
    got = backend.gemm_epilogue(a, b, lhs_transposed=lt, rhs_transposed=rt, out_dtype=torch.float32)
    torch.cuda.synchronize()
    backend.poll()
    want = (a.double().t() if lt else a.double()) @ (b.double().t() if rt else b.double())
    # products are exact in f32; a chain of k of them of magnitude <= 1 is off by at most k * 2^-24 * sum |a b| <= k^2 * 2^-24,
    # and by about sqrt(k) * 2^-24 * sqrt(k) in the mean: 64 times the mean
    assert (got.double() - want).abs().max().item() <= 64 * max(k, 64) * 2.0 ** -24


@pytest.mark.parametrize("epilogue", [abi.EPI_NONE, abi.EPI_BIAS, abi.EPI_BIAS_GELU, abi.EPI_SWIGLU])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m,n,k", [(8, 96, 520), (40, 608, 256), (200, 4128, 128)])
def test_rows_do_not_depend_on_the_batch(backend, epilogue, out_dtype, m, n, k):
    if epilogue == abi.EPI_SWIGLU and out_dtype == torch.float32:
        pytest.skip("SwiGLU narrows")
    rows = 4096   # the pair kernel's side of the rule
    a, b = operands(rows, n, k, torch.bfloat16, False, False)
    bias = torch.linspace(-1, 1, n, device="cuda") if epilogue in (abi.EPI_BIAS, abi.EPI_BIAS_GELU) else None
    whole = backend.gemm_epilogue(a, b, bias, epilogue=epilogue, out_dtype=out_dtype)
    part = backend.gemm_epilogue(a[:m].contiguous(), b, bias, epilogue=epilogue, out_dtype=out_dtype)
    torch.cuda.synchronize()
    backend.poll()
    assert torch.equal(part.view(torch.uint8), whole[:m].contiguous().view(torch.uint8))


@pytest.mark.parametrize("k", [1016, 1024, 1032, 1088, 1096, 1152, 1216, 1280, 1288, 2056, 4096])
@pytest.mark.parametrize("rt", [False, True])
@pytest.mark.parametrize("m,n", [(8, 72), (16, 192)])
def test_stages_of_four_blocks_are_exact_on_integers(backend, m, n, k, rt):
    # Rings of at least eight stages are walked four 64-element blocks of K at a time: whole and ragged last stages and last
    # blocks. Sums of products of small integers are exact in f32, so the result is.
    gen = torch.Generator(device="cuda").manual_seed(k)
    a = torch.randint(-4, 5, (m, k), device="cuda", generator=gen).bfloat16()
    b = torch.randint(-4, 5, (n, k) if rt else (k, n), device="cuda", generator=gen).bfloat16()
    out = backend.gemm_epilogue(a, b, rhs_transposed=rt, out_dtype=torch.float32)
    torch.cuda.synchronize()
    backend.poll()
    assert torch.equal(out.double(), a.double() @ (b.double().T if rt else b.double()))
