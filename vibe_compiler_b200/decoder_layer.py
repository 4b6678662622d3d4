"""Llama-style decoder layer (RMSNorm, RoPE, grouped-query causal attention, SwiGLU FFN) on the B200
backend, tensor-parallel over heads and FFN columns with one all-reduce after the output projection
and one after the down projection.

The reference lowers such a block to GEMM / attention / elementwise command regions for its 16 Tiles
and realises the two sums with ring or recursive-doubling collectives over the on-chip network
(lib/Wafer/Transforms/Tile/DistributedCollectiveMovement.cpp:675-735); here each region is one
library kernel and the sums are done by the NVSwitch through the library's multimem kernel (sharding.SwitchSum;
torch symmetric memory supplies the multicast-bound buffers), or by torch.distributed's all-reduce where the GPUs
offer no NVLink multicast.

Sharding (rank r of G): query heads [r*Hq/G, (r+1)*Hq/G), KV heads likewise, FFN columns likewise.
RMSNorm and the residual adds are replicated. Every GEMM, the attention, the norms, RoPE and the adds
run in libwb200 kernels; nothing is computed by PyTorch.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Optional

import torch

from . import _abi as abi
from .backend import B200TargetModelBackend


@dataclass
class LayerConfig:
    d_model: int = 4096
    q_heads: int = 32
    kv_heads: int = 8
    head_dim: int = 128
    ffn: int = 14336
    eps: float = 1e-5
    rope_theta: float = 10000.0


@dataclass
class LayerWeights:
    """Full (unsharded) weights, [in, out] row-major, in the storage dtype."""
    norm1: torch.Tensor   # [d_model]
    wq: torch.Tensor      # [d_model, q_heads * head_dim]
    wk: torch.Tensor      # [d_model, kv_heads * head_dim]
    wv: torch.Tensor      # [d_model, kv_heads * head_dim]
    wo: torch.Tensor      # [q_heads * head_dim, d_model]
    norm2: torch.Tensor   # [d_model]
    wgate: torch.Tensor   # [d_model, ffn]
    wup: torch.Tensor     # [d_model, ffn]
    wdown: torch.Tensor   # [ffn, d_model]


def random_weights(cfg: LayerConfig, dtype=torch.bfloat16, seed: int = 20260803, std: float = 0.02) -> LayerWeights:
    g = torch.Generator(device="cpu").manual_seed(seed)

    def w(*shape):
        return (torch.randn(*shape, generator=g) * std).to(dtype)
    hd = cfg.head_dim
    return LayerWeights(
        norm1=(1.0 + torch.randn(cfg.d_model, generator=g) * std).to(dtype),
        wq=w(cfg.d_model, cfg.q_heads * hd), wk=w(cfg.d_model, cfg.kv_heads * hd), wv=w(cfg.d_model, cfg.kv_heads * hd),
        wo=w(cfg.q_heads * hd, cfg.d_model),
        norm2=(1.0 + torch.randn(cfg.d_model, generator=g) * std).to(dtype),
        wgate=w(cfg.d_model, cfg.ffn), wup=w(cfg.d_model, cfg.ffn), wdown=w(cfg.ffn, cfg.d_model))


class ShardedDecoderLayer:
    """One rank's shard of the layer. `group` is a torch.distributed process group (None: single GPU)."""

    def __init__(self, backend: B200TargetModelBackend, cfg: LayerConfig, weights: LayerWeights, rank: int = 0,
                 world_size: int = 1, group=None, device: Optional[torch.device] = None):
        if cfg.q_heads % world_size or cfg.kv_heads % world_size or cfg.ffn % world_size:
            raise ValueError("heads and FFN width must divide by the world size")
        if (cfg.ffn // world_size) % 16:
            raise ValueError("FFN columns per rank must be a multiple of 16 (interleaved SwiGLU epilogue)")
        self.backend, self.cfg, self.rank, self.world, self.group = backend, cfg, rank, world_size, group
        device = device or torch.device("cuda", backend.device)
        hd = cfg.head_dim
        self.hq, self.hkv, self.ffn = cfg.q_heads // world_size, cfg.kv_heads // world_size, cfg.ffn // world_size
        q0, k0, f0 = rank * self.hq * hd, rank * self.hkv * hd, rank * self.ffn
        # fused QKV projection: columns [q heads | k heads | v heads] of this rank
        self.wqkv = torch.cat([weights.wq[:, q0:q0 + self.hq * hd], weights.wk[:, k0:k0 + self.hkv * hd],
                               weights.wv[:, k0:k0 + self.hkv * hd]], dim=1).contiguous().to(device)
        self.wo = weights.wo[q0:q0 + self.hq * hd].contiguous().to(device)
        # gate and up columns interleaved so the GEMM epilogue sees (gate_j, up_j) side by side
        gate, up = weights.wgate[:, f0:f0 + self.ffn], weights.wup[:, f0:f0 + self.ffn]
        self.wgu = torch.stack([gate, up], dim=2).reshape(cfg.d_model, 2 * self.ffn).contiguous().to(device)
        self.wdown = weights.wdown[f0:f0 + self.ffn].contiguous().to(device)
        self.norm1, self.norm2 = weights.norm1.to(device), weights.norm2.to(device)

    def _all_reduce(self, tensor):
        if self.world > 1:
            import torch.distributed as dist
            dist.all_reduce(tensor, op=dist.ReduceOp.SUM, group=self.group)
        return tensor

    def attention_partial(self, tokens: torch.Tensor, batch: int, seq: int, position_offset: int = 0) -> torch.Tensor:
        """This rank's share of the attention block output (before the sum over head shards): [tokens, d_model]."""
        be, cfg = self.backend, self.cfg
        h = be.rmsnorm(tokens, self.norm1, cfg.eps)
        qkv = be.gemm_epilogue(h, self.wqkv)
        q, k, v = be.rope_split(qkv, batch, seq, self.hq, self.hkv, cfg.head_dim, cfg.rope_theta, position_offset)
        attn = be.attention_fa(q, k, v, cfg.head_dim ** -0.5, True, token_major_out=True)      # [batch, seq, hq, hd]
        return be.gemm_epilogue(attn.reshape(batch * seq, self.hq * cfg.head_dim), self.wo)

    def ffn_partial(self, x1: torch.Tensor) -> torch.Tensor:
        """This rank's share of the FFN output (before the sum over FFN shards): [tokens, d_model]."""
        be, cfg = self.backend, self.cfg
        h2 = be.rmsnorm(x1, self.norm2, cfg.eps)
        act = be.gemm_epilogue(h2, self.wgu, epilogue=abi.EPI_SWIGLU)                          # [tokens, ffn / G]
        return be.gemm_epilogue(act, self.wdown)

    def forward(self, x: torch.Tensor, position_offset: int = 0) -> torch.Tensor:
        """x: [batch, seq, d_model] on this rank's GPU (replicated across ranks). Returns the layer output."""
        batch, seq, d = x.shape
        tokens = x.reshape(batch * seq, d)
        partial = self._all_reduce(self.attention_partial(tokens, batch, seq, position_offset))   # sum over head shards
        x1 = self.backend.residual_add(tokens, partial)
        partial2 = self._all_reduce(self.ffn_partial(x1))                                         # sum over FFN shards
        return self.backend.residual_add(x1, partial2).reshape(batch, seq, d)


    def default_micro_batches(self, batch: int) -> int:
        """Parts the batch is cut into so that the sums of one part travel while the next computes. More parts hide more of
        the communication but shrink the per-part GEMMs, which costs more the narrower the shard (measured on 8 GPUs: the
        kernels alone take 0.93 / 1.05 / 1.3 ms with 1 / 2 / 4 parts): 2 parts."""
        if self.world == 1:
            return 1
        return 2 if batch % 2 == 0 else 1

    def default_reserved_sms(self) -> int:
        """SMs the persistent kernels leave to the sums. The library's switch kernel moves a rank's slice (1 / world of the
        buffer) at the link's rate from two or four SMs (measured: 4 SMs on 8 GPUs, 8 on 2 - fewer halve its rate, more
        only take SMs from the GEMMs); NCCL wants more (measured best: 24 on 8 GPUs, 16 on 2)."""
        if self.world == 1:
            return 0
        if self.switch_sums() is not None:
            return 4 if self.world >= 8 else 8
        return 24 if self.world >= 8 else 16

    def forward_fused(self, x: torch.Tensor, position_offset: int = 0, micro_batches: Optional[int] = None,
                      reserved_sms: Optional[int] = None) -> torch.Tensor:
        """Same computation through the single C-ABI call (wb200_decoder_layer): nine kernels per part enqueued by one call,
        the two sums through a callback into torch.distributed, intermediates in one reused workspace. With several
        shards the batch is cut into `micro_batches` parts whose sums run on a second stream while the following parts
        compute; `reserved_sms` SMs stay free for the sum's kernel. The sums are done by the NVSwitch through the
        library's own kernel (switch_sums()) where the GPUs offer NVLink multicast, else by torch.distributed."""
        reduce, factory, native = None, None, None
        reserved = reserved_sms if reserved_sms is not None else self.default_reserved_sms()
        if self.world > 1:
            import torch.distributed as dist
            sums = self.switch_sums(blocks=reserved)
            if sums is not None:
                factory = sums.allocate
            if not getattr(self, "_all_reduce_enabled", True):   # timing aid: the layer's kernels without the sums (wrong values)
                reduce = lambda t: None                # noqa: E731
            elif sums is not None:
                native = sums                          # the library launches its own sum kernel: no callback into Python
            else:
                reduce = lambda t: dist.all_reduce(t, op=dist.ReduceOp.SUM, group=self.group)   # noqa: E731
        out, self._workspace = self.backend.decoder_layer(
            x, norm1=self.norm1, wqkv=self.wqkv, wo=self.wo, norm2=self.norm2, wgu=self.wgu, wdown=self.wdown, q_heads=self.hq,
            kv_heads=self.hkv, head_dim=self.cfg.head_dim, eps=self.cfg.eps, rope_theta=self.cfg.rope_theta,
            position_offset=position_offset, allreduce=reduce, workspace=getattr(self, "_workspace", None),
            micro_batches=(micro_batches if micro_batches is not None else self.default_micro_batches(x.shape[0])),
            reserved_sms=reserved, workspace_factory=factory, switch_sum=native)
        return out

    def switch_sums(self, blocks: int = 0):
        """The NVSwitch sum of this layer's group (sharding.SwitchSum), made on first use by a collective call, or None:
        one shard, no multicast on these GPUs, or WB200_LAYER_SUM=nccl in the environment (the library all-reduce)."""
        import os
        if self.world == 1 or os.environ.get("WB200_LAYER_SUM", "switch") == "nccl":
            return None
        if not hasattr(self, "_switch_sums"):
            from .sharding import SwitchSum
            try:
                sums = SwitchSum(self.backend, self.group, blocks=blocks)
                self._switch_sums = sums if sums.available else None
            except (RuntimeError, AttributeError):      # symmetric memory or multicast unavailable in this process
                self._switch_sums = None
            self._workspace = None                      # the workspace has to be symmetric from now on
        if self._switch_sums is not None:
            self._switch_sums.blocks = blocks
        return self._switch_sums


def layer_flops(cfg: LayerConfig, batch: int, seq: int) -> int:
    """Algorithmic flop of one forward pass (causal attention counts visible pairs only)."""
    t = batch * seq
    hd = cfg.head_dim
    gemm = 2 * t * cfg.d_model * ((cfg.q_heads + 2 * cfg.kv_heads) * hd + cfg.q_heads * hd + 3 * cfg.ffn)
    attention = 4 * batch * cfg.q_heads * hd * seq * (seq + 1) // 2
    return gemm + attention
