"""Wide & Deep on sharded sparse tables.

``WideAndDeep``: single-hot categorical fields; the wide part is a dim-1
embedding per id (summed), the deep part a dim-``dim`` embedding per field
concatenated with the dense features and fed to an MLP - the structure of the
reference's example (examples/WideAndDeep/model.py:60-125), with the hashed
one-hot wide features expressed as a dim-1 table.

``MultiHotWideAndDeep``: every field is a bag of ids (JaggedTensor); all
fields share one combined table keyed by a 64-bit hash, pooled by sum or mean
per field.  On the GPU engine each lookup is one fused pull (dedup, exchange,
gather and pooling) and one fused push.
"""
from __future__ import annotations

from typing import List, Sequence

import torch
from torch.nn.modules.module import _has_any_global_hook

from .. import pytorch as kk
from .._native import C
from ..ops import counters
from .mlp import MLP


class WideAndDeep(torch.nn.Module):
    def __init__(self, num_fields: int = 26, num_dense: int = 13, dim: int = 8, hidden: Sequence[int] = (256, 128),
                 name: str = "wide_deep", combine: bool = False):
        """``combine``: both tables go through one ``CombineEmbedding`` - one request round per step and direction
        instead of two (what counts on the TCP deployment, where a round is a message to every server)."""
        super().__init__()
        self.num_fields, self.num_dense, self.dim = num_fields, num_dense, dim
        if combine:
            self.both = kk.CombineEmbedding([1, dim], initializers=[kk.ConstantInitializer(0.0),
                                                                    kk.NormalInitializer(0.0, 0.05)],
                                            names=[f"{name}.wide", f"{name}.deep"])
        else:
            self.both = None
            self.wide = kk.Embedding(1, initializer=kk.ConstantInitializer(0.0), name=f"{name}.wide")
            self.deep = kk.Embedding(dim, initializer=kk.NormalInitializer(0.0, 0.05), name=f"{name}.deep")
        width = num_fields * dim + num_dense
        self.mlp_in = (width + 7) // 8 * 8
        self.mlp = MLP(self.mlp_in, list(hidden) + [1])
        self.bias = torch.nn.Parameter(torch.zeros(1))

    def forward(self, dense: torch.Tensor, ids: torch.Tensor) -> torch.Tensor:
        if self.both is not None:
            w, e = self.both([ids, ids])
            wide = w.sum(dim=(1, 2))
        elif self._fused_ok(dense, ids):
            prepared = self.mlp.prepare()  # weight casts run beside the sparse pull
            x, wide = _WideDeepFront.apply(self.deep.sparse_table, self.wide.sparse_table, dense, ids, self.mlp_in, self.dim)
            return self.mlp(x, input_grad_cols=self.num_fields * self.dim, addend=wide,
                            prepared=prepared).squeeze(-1) + self.bias
        else:
            wide = self.wide(ids).sum(dim=(1, 2))
            e = self.deep(ids)
        dense = dense.to(e.device)
        parts = [e.flatten(1), dense]
        if self.mlp_in > e.shape[1] * e.shape[2] + dense.shape[1]:
            parts.append(torch.zeros(dense.shape[0], self.mlp_in - e.shape[1] * e.shape[2] - dense.shape[1],
                                     dtype=e.dtype, device=e.device))
        return wide + self.mlp(torch.cat(parts, dim=1)).squeeze(-1) + self.bias

    def _fused_ok(self, dense: torch.Tensor, ids: torch.Tensor) -> bool:
        """Whether one dedup and one kernel can stand for the two lookups, their sum and the concatenation: one GPU, the
        stock modules without hooks, tables that are float32 and trained alike, and a float32 batch without gradient."""
        from ..pytorch import native
        if not ids.is_cuda or ids.dim() != 2 or ids.shape[1] != self.num_fields or not native.is_initialized():
            return False
        eng = native.engine()
        chunks = self.dim // 4
        tables = (self.wide.sparse_table, self.deep.sparse_table)
        return (hasattr(eng, "pull_sparse_unique") and eng.world == 1 and not eng.cfg.long_id_streams
                and self.dim % 4 == 0 and chunks & (chunks - 1) == 0 and self.dim <= 128
                and all(_stock(m, kk.Embedding) for m in (self.wide, self.deep)) and _stock_mlp(self.mlp)
                and all(t.dtype() == torch.float32 and t.table_id() is not None
                        and (t.requires_grad or not torch.is_grad_enabled()) for t in tables)
                and dense.dtype == torch.float32 and not dense.requires_grad and dense.dim() == 2
                and dense.shape[0] == ids.shape[0] and dense.shape[1] <= self.mlp_in - self.num_fields * self.dim)


def _stock(module, cls) -> bool:
    """Whether calling ``module`` runs ``cls.forward`` and nothing else: the class itself, no hooks."""
    return (type(module) is cls and "forward" not in vars(module) and not module._forward_pre_hooks
            and not module._forward_hooks and not module._backward_hooks and not module._backward_pre_hooks
            and not _has_any_global_hook())


def _stock_mlp(mlp) -> bool:
    """Whether ``mlp`` takes a bfloat16 input as it takes the float32 one that it would round."""
    return _stock(mlp, MLP) and mlp.use_tensor_cores and mlp.layers[0].weight.is_cuda


class _WideDeepFront(torch.autograd.Function):
    """Both lookups with one dedup -> pack kernel -> (bf16 MLP input, sum of the wide weights); the backward kernel adds
    every occurrence's gradient into the push buffers.  What DeepFM's front end does, without the second-order term.  Of the
    38 kernels of a step by modules, a dozen moved the rows from one to the next."""

    @staticmethod
    def forward(ctx, deep_table, wide_table, dense, ids, width, dim):
        from ..pytorch import native
        eng = native.engine()
        id2, id1 = deep_table.table_id(), wide_table.table_id()
        B, F = ids.shape
        in_place = ids.numel() <= (1 << 19)  # as DeepFM
        rows2, inv2, t2 = eng.pull_sparse_unique(id2, ids, in_place=in_place)
        rows1, inv1, t1 = eng.pull_sparse_unique(id1, ids, share_with=id2, in_place=in_place)
        x = torch.empty((B, width), dtype=torch.bfloat16, device=rows2.device)
        wide = torch.empty(B, dtype=torch.float32, device=rows2.device)
        dense = dense.to(rows2.device).contiguous()
        counters.add()
        C.deepfm_pack_forward(rows2, inv2, rows1, inv1, dense, B, F, dim, x, wide, t2.slots, t1.slots, fm=False)
        ctx.state = (eng, id1, id2, rows2, inv2, inv1, t1, t2, dim, ids)
        return x, wide

    @staticmethod
    def backward(ctx, dx, dwide):
        eng, id1, id2, rows2, inv2, inv1, t1, t2, dim, ids = ctx.state
        B, F = ids.shape
        dwide = dwide.float().contiguous()
        if not (t1.current(eng.channels[id1]) and t2.current(eng.channels[id2])):
            # another lookup has used the channels since: the gradients go out by id
            eng.push_sparse_table(id2, ids, dx[:, :F * dim].float().reshape(B, F, dim))
            eng.push_sparse_table(id1, ids, dwide.view(B, 1, 1).expand(B, F, 1).contiguous())
            return None, None, None, None, None, None
        counters.add()
        C.deepfm_pack_backward(rows2, inv2, inv1, dx.contiguous(), dwide, B, F, dim, eng.grad_accumulator(id2),
                               eng.grad_accumulator(id1), t2.slots, None)
        eng.push_sparse_accumulated(id1, t1)
        eng.push_sparse_accumulated(id2, t2)
        return None, None, None, None, None, None


class MultiHotWideAndDeep(torch.nn.Module):
    """``forward(dense, bags)`` with ``bags`` = one JaggedTensor whose bags are laid out
    sample-major, field-minor: bag ``b * num_fields + f`` holds sample b's ids of field f."""

    def __init__(self, num_fields: int = 100, num_dense: int = 13, dim: int = 64,
                 hidden: Sequence[int] = (1024, 512, 256), mean_fields: Sequence[int] = (), name: str = "mh_wide_deep"):
        super().__init__()
        self.num_fields, self.num_dense, self.dim = num_fields, num_dense, dim
        self.wide = kk.JaggedEmbedding(1, initializer=kk.ConstantInitializer(0.0), name=f"{name}.wide", mode="sum")
        self.deep = kk.Embedding(dim, initializer=kk.NormalInitializer(0.0, 0.05), name=f"{name}.combined")
        mean = torch.zeros(num_fields, dtype=torch.uint8)
        if len(mean_fields):
            mean[list(mean_fields)] = 1
        self.register_buffer("field_is_mean", mean)
        width = num_fields * dim + num_dense
        self.mlp_in = (width + 7) // 8 * 8
        self.mlp = MLP(self.mlp_in, list(hidden) + [1])
        self.bias = torch.nn.Parameter(torch.zeros(1))

    def forward(self, dense: torch.Tensor, bags: kk.JaggedTensor) -> torch.Tensor:
        from ..pytorch import native

        k = bags.num_bags()
        B = k // self.num_fields
        wide = self.wide(bags).view(B, self.num_fields).sum(1)
        eng = native.engine()
        if hasattr(eng, "pull_sparse_pooled"):
            # both tables look the same ids up: where the wide one's lookup is known to be that, its dedup serves both
            share = self.wide.embedding.sparse_table.table_id() if self._wide_is_one_lookup(bags) else None
            if self._pools_into_mlp(eng, dense, B):
                x = _PooledInput.apply(self.deep.sparse_table, bags.values(), bags.offsets(), self.field_is_mean.repeat(B),
                                       dense, self.num_fields, self.mlp_in, share)
                return wide + self.mlp(x, input_grad_cols=self.num_fields * self.dim).squeeze(-1) + self.bias
            pooled = _PooledLookup.apply(self.deep.sparse_table, bags.values(), bags.offsets(),
                                         self.field_is_mean.repeat(B), share)
        else:
            emb = self.deep(bags.values())
            off = bags.offsets()
            s = native.jagged_sum_forward(emb, off, 0.0)  # plain CPU path: sum, then scale the mean fields
            lens = (off[1:] - off[:-1]).clamp(min=1).to(s.dtype).unsqueeze(1)
            is_mean = self.field_is_mean.repeat(B).bool().unsqueeze(1)
            pooled = _CpuPool.apply(emb, off, is_mean, lens)
        dense = dense.to(pooled.device)
        parts = [pooled.view(B, self.num_fields * self.dim), dense]
        pad = self.mlp_in - self.num_fields * self.dim - dense.shape[1]
        if pad:
            parts.append(torch.zeros(B, pad, dtype=pooled.dtype, device=pooled.device))
        return wide + self.mlp(torch.cat(parts, dim=1)).squeeze(-1) + self.bias

    def _pools_into_mlp(self, eng, dense: torch.Tensor, samples: int) -> bool:
        """Whether the lookup can write the MLP's input itself: what stands between them is the stock module without
        hooks on the tensor cores, and nothing else wants the float32 input or its gradient."""
        return (hasattr(eng, "pools_into_input") and eng.pools_into_input(self.deep.sparse_table.table_id())
                and _stock_mlp(self.mlp) and dense.dtype == torch.float32 and not dense.requires_grad and dense.dim() == 2
                and dense.shape[0] == samples and dense.shape[1] <= self.mlp_in - self.num_fields * self.dim)

    def _wide_is_one_lookup(self, bags: kk.JaggedTensor) -> bool:
        """Whether calling ``self.wide`` on ``bags`` has been one fused lookup of exactly their ids, with nothing behind
        it: the module as it was made, without hooks that might change the ids or look others up, on the fused path."""
        w = self.wide
        return (type(w) is kk.JaggedEmbedding and type(w.embedding) is kk.Embedding and "forward" not in vars(w)
                and not w._forward_pre_hooks and not w._forward_hooks and not _has_any_global_hook()
                and w.fused(bags))


class _PooledInput(torch.autograd.Function):
    """Fused bag lookup that ends in the bfloat16 input of the MLP: pooled rows, dense features, zeros (one GPU).  The
    MLP would round its input to bfloat16 and hands back a bfloat16 gradient in any case; as float32 both crossed memory
    three times more, in a concatenation and conversions (4096 samples of 100 fields x 64: 210 us of a step of 2800)."""

    @staticmethod
    def forward(ctx, sparse_table, values, offsets, bag_mean, dense, fields, width, share_with):
        from ..pytorch import native
        eng = native.engine()
        tid = sparse_table.table_id()
        x, ticket = eng.pull_sparse_input(tid, values, offsets, bag_mean, dense, fields, width, share_with=share_with)
        ctx.state = (eng, tid, ticket, values, fields)
        return x

    @staticmethod
    def backward(ctx, grad):
        eng, tid, ticket, values, fields = ctx.state
        eng.push_sparse_pooled(tid, ticket, grad, values, fields=fields)
        return None, None, None, None, None, None, None, None


class _PooledLookup(torch.autograd.Function):
    """Fused bag lookup with a per-bag sum / mean switch (GPU engine).  ``share_with``: id of a table that has just
    looked the same ids up, whose dedup is used again."""

    @staticmethod
    def forward(ctx, sparse_table, values, offsets, bag_mean, share_with):
        from ..pytorch import native
        eng = native.engine()
        tid = sparse_table.table_id()
        out, ticket = eng.pull_sparse_pooled(tid, values, offsets, bag_mean=bag_mean, share_with=share_with)
        ctx.state = (eng, tid, ticket, values)
        return out

    @staticmethod
    def backward(ctx, grad):
        eng, tid, ticket, values = ctx.state
        eng.push_sparse_pooled(tid, ticket, grad.contiguous(), values)
        return None, None, None, None, None


class _CpuPool(torch.autograd.Function):
    @staticmethod
    def forward(ctx, emb, offsets, is_mean, lens):
        from ..pytorch import native
        ctx.save_for_backward(offsets, is_mean, lens)
        s = native.jagged_sum_forward(emb, offsets, 0.0)
        return torch.where(is_mean, s / lens, s)

    @staticmethod
    def backward(ctx, grad):
        from ..pytorch import native
        offsets, is_mean, lens = ctx.saved_tensors
        g = torch.where(is_mean, grad / lens, grad).contiguous()
        return native.jagged_sum_backward(offsets, g), None, None, None
