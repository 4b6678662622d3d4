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


@pytest.mark.parametrize("d_model", [128, 2056, 8320])
def test_layer_with_the_add_inside_the_norm(backend, d_model):
    # the fused layer adds the residual inside the second norm; the same layer from separate kernels has the same bits
    # (rows below, at and beyond what the norm keeps in registers)
    from vibe_compiler_b200.decoder_layer import LayerConfig, LayerWeights, ShardedDecoderLayer
    cfg = LayerConfig(d_model=d_model, q_heads=2, kv_heads=1, ffn=256)
    gen = torch.Generator(device="cuda").manual_seed(d_model)
    w = lambda *shape: (torch.randn(shape, device="cuda", generator=gen) * 0.02).bfloat16()
    hd = cfg.head_dim
    weights = LayerWeights(norm1=1 + w(d_model), wq=w(d_model, 2 * hd), wk=w(d_model, hd), wv=w(d_model, hd), wo=w(2 * hd, d_model),
                           norm2=1 + w(d_model), wgate=w(d_model, 256), wup=w(d_model, 256), wdown=w(256, d_model))
    layer = ShardedDecoderLayer(backend, cfg, weights)
    x = torch.randn(2, 36, d_model, device="cuda", generator=gen).bfloat16()
    fused, separate = layer.forward_fused(x), layer.forward(x)
    torch.cuda.synchronize()
    backend.poll()
    assert torch.equal(fused, separate)


@pytest.mark.parametrize("seq", [32, 136])
def test_parts_with_kept_sms_equal_one_pass(backend, seq):
    """Parts of few tokens with SMs kept for the sums: the gate/up projection has more tiles than SMs to use and goes to CTA pairs of
    which the rows fill a part, where one pass takes the tile kernel. The bits are the same."""
    from vibe_compiler_b200.decoder_layer import LayerConfig, ShardedDecoderLayer, random_weights
    cfg = LayerConfig(d_model=512, q_heads=4, kv_heads=2, ffn=14336)
    layer = ShardedDecoderLayer(backend, cfg, random_weights(cfg))
    x = torch.randn(2, seq, cfg.d_model, generator=torch.Generator().manual_seed(seq)).bfloat16().cuda()
    kwargs = dict(norm1=layer.norm1, wqkv=layer.wqkv, wo=layer.wo, norm2=layer.norm2, wgu=layer.wgu, wdown=layer.wdown, q_heads=layer.hq,
                  kv_heads=layer.hkv, head_dim=cfg.head_dim, eps=cfg.eps, rope_theta=cfg.rope_theta, allreduce=lambda tensor: None)
    one, _ = backend.decoder_layer(x, **kwargs)
    for reserved in (4, 16):
        parts, _ = backend.decoder_layer(x, micro_batches=2, reserved_sms=reserved, **kwargs)
        torch.cuda.synchronize()
        backend.poll()
        assert torch.equal(one, parts)
