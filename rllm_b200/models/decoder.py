"""The generic decoder: any ``ModelSpec`` built from registered parts.

This is the only model class of the framework.  An architecture is a function
from its typed configuration to a ``ModelSpec``; the decoder builds the parts
the spec names, collects the tensors they declare, works out which runs of the
order need which kind of cache, and runs a step:

    embedding -> for each run of the order: block(run.layer) with the cache of
    run.cache -> final norm on the rows that were asked for -> head.

(The reference's forward is the fixed loop of crates/rllm-model/src/llama.rs:283-326,
with the head applied to every row at :70.)
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Dict, List, Optional, Sequence, Tuple

import torch

from ..parts import registry as part_registry
from ..parts.base import KVCacheView, PendingSum, StateCacheView, StepContext
from ..parts.embedding import OutputHead, TokenEmbedding
from ..parts.spec import KVPagesNeed, ModelSpec, StateNeed, TensorSpec
from ..weights.loader import WeightSource, load_tensors


@dataclass
class CacheLayout:
    """groups[g]: the need shared by the runs of group g.  owners[g]: the runs
    (indices into the order) that own storage in group g.  run_group[i] and
    run_owner[i]: the group of run i and the run whose storage it uses (None:
    the run's mixer keeps nothing)."""

    groups: List[object]
    owners: List[list]
    run_group: List[object]
    run_owner: List[Optional[int]]


class DecoderModel:
    def __init__(self, spec: ModelSpec):
        spec.validate()
        self.spec = spec
        self.embedding = TokenEmbedding(spec.embedding)
        self.blocks = []
        for ls in spec.layers:
            mixer = part_registry.build_part("mixer", ls.mixer, prefix=ls.prefix + _sub(ls.mixer))
            ffn = None if ls.ffn is None else \
                part_registry.build_part("feed_forward", ls.ffn, prefix=ls.prefix + _sub(ls.ffn))
            norms = [part_registry.build_part("norm", n, prefix=ls.prefix) for n in ls.norms]
            if ls.block not in part_registry.BLOCKS:
                raise KeyError(f"no block arrangement {ls.block!r}; known: {sorted(part_registry.BLOCKS)}")
            if ls.block_params is not None:
                # an arrangement with sizes, constants and tensors of its own
                self.blocks.append(part_registry.BLOCKS[ls.block](mixer, ffn, norms, spec=ls.block_params,
                                                                  prefix=ls.prefix))
            else:
                self.blocks.append(part_registry.BLOCKS[ls.block](mixer, ffn, norms))
        self.final_norm = part_registry.build_part("norm", spec.final_norm)
        self.head = OutputHead(spec.head)
        self.layout = self._cache_layout()
        # blocks whose stream is a weighted sum of all earlier results: how many results the model keeps
        self.depth_levels = max((int(getattr(b, "depth_levels", 0) or 0) for b in self.blocks), default=0)
        self.dtype: Optional[torch.dtype] = None
        self.device: Optional[torch.device] = None

    # -- weights ----------------------------------------------------------
    def parts(self):
        out = [self.embedding]
        for b in self.blocks:
            out.extend(b.parts())
        out += [self.final_norm, self.head]
        return out

    def tensor_specs(self) -> List[TensorSpec]:
        seen: Dict[str, TensorSpec] = {}
        for part in self.parts():
            for ts in part.tensor_specs():
                if ts.name in seen and seen[ts.name].shape != ts.shape:
                    raise ValueError(f"tensor {ts.name!r} is declared twice with different shapes")
                seen.setdefault(ts.name, ts)
        return list(seen.values())

    def load(self, source: WeightSource, run_dtype: torch.dtype, device: torch.device) -> None:
        ignored = [n for part in self.parts() for n in part.ignored_tensors()]
        tensors = load_tensors(self.tensor_specs(), source, run_dtype, device, ignored)
        for part in self.parts():
            part.load(tensors)
        self.dtype, self.device = run_dtype, device

    def num_weight_bytes(self) -> int:
        spans = sorted((v.data_ptr(), v.data_ptr() + v.numel() * v.element_size())
                       for part in self.parts() for v in vars(part).values() if isinstance(v, torch.Tensor))
        total = end = 0
        for a, b in spans:                       # (a part may keep a tensor and a view of it)
            total += max(0, b - max(a, end))
            end = max(end, b)
        return total

    def step_scratch(self) -> int:
        """Bytes that a step may take by what the cache holds; layers run one after the other."""
        return max((b.mixer.step_scratch() for b in self.blocks), default=0)

    # -- cache ------------------------------------------------------------
    def _cache_layout(self) -> CacheLayout:
        groups: List[object] = []
        owners: List[list] = []
        run_group: List[object] = []
        run_owner: List[Optional[int]] = []

        def needs_of(run) -> Tuple[Tuple[object, ...], bool]:
            need = self.blocks[run.layer].mixer.cache_need()
            if need is None:
                return (), False
            return (tuple(need), True) if isinstance(need, (tuple, list)) else ((need,), False)

        for i, run in enumerate(self.spec.order):
            needs, several = needs_of(run)
            if not needs:
                run_group.append(None)
                run_owner.append(None)
                continue
            # a slot keeps what its owner and every run that reads it need: the same rows, the widest window
            needs = list(needs)
            for j, other in enumerate(self.spec.order):
                if other.cache != run.cache or j == i:
                    continue
                theirs, _ = needs_of(other)
                if len(theirs) != len(needs):
                    raise ValueError(f"order[{i}] and order[{j}] use cache slot {run.cache} but keep "
                                     f"{needs} and {list(theirs)}")
                for k, (mine, other_need) in enumerate(zip(needs, theirs)):
                    wide = mine.widened(other_need) if hasattr(mine, "widened") and type(other_need) is type(mine) \
                        else (mine if other_need == mine else None)
                    if wide is None:
                        raise ValueError(f"order[{i}] and order[{j}] use cache slot {run.cache} but keep "
                                         f"{mine} and {other_need}")
                    needs[k] = wide
            gs = []
            for k, need in enumerate(needs):
                if need not in groups:
                    groups.append(need)
                    owners.append([])
                g = groups.index(need)
                if run.cache == i:
                    owners[g].append((i, k) if several else i)
                gs.append(g)
            run_group.append(tuple(gs) if several else gs[0])
            run_owner.append(run.cache)
        return CacheLayout(groups, owners, run_group, run_owner)

    # -- compute ----------------------------------------------------------
    def forward(self, token_ids: torch.Tensor, ctx: StepContext, logit_rows: torch.Tensor,
                storage) -> torch.Tensor:
        """Logits float32 [R, vocab] at the rows ``logit_rows`` (int32 indices
        into this step's tokens).  ``storage.view(run_index)`` gives a run's
        cache view."""
        if self.depth_levels:
            # level 0 is the embedding's output, level i + 1 the result of run i; the blocks fill and read it
            hist = torch.empty((self.depth_levels, token_ids.numel(), self.spec.hidden_size), dtype=torch.float32,
                               device=token_ids.device)
            ctx.extras["depth_history"] = hist
            h = self.embedding.forward(token_ids, ctx.err, out=hist[0])
        elif self.spec.streams > 0:
            # several copies of the residual, all equal to the embedding's output at the start
            h = torch.empty((self.spec.streams, token_ids.numel(), self.spec.hidden_size), dtype=torch.float32,
                            device=token_ids.device)
            self.embedding.forward(token_ids, ctx.err, out=h)
        else:
            h = self.embedding.forward(token_ids, ctx.err)
        pending = None
        order = self.spec.order
        for i, run in enumerate(order):
            block = self.blocks[run.layer]
            if getattr(block, "takes_next_block", False):
                # the block that reads the streams next: this one may prepare its input in its last kernel
                nxt = self.blocks[order[i + 1].layer] if i + 1 < len(order) else None
                h, pending = block.forward(h, pending, ctx, storage.view(i), next_block=nxt)
            elif getattr(block, "takes_next_norm", False) and i + 1 < len(order):
                # the norm that reads the stream after this block: the block may prepare its input
                nxt = getattr(self.blocks[order[i + 1].layer], "norms", None)
                h, pending = block.forward(h, pending, ctx, storage.view(i), next_norm=nxt[0] if nxt else None)
            elif getattr(block, "takes_final_norm", False) and self.spec.streams == 0:
                # the last block, and one that wants to know: the model's own norm reads the stream next
                h, pending = block.forward(h, pending, ctx, storage.view(i), next_norm=self.final_norm)
            else:
                h, pending = block.forward(h, pending, ctx, storage.view(i))
        if logit_rows.numel() == 0:
            return torch.empty((0, self.spec.vocab_size), dtype=torch.float32, device=h.device)
        if not isinstance(pending, torch.Tensor) and not (
                isinstance(pending, PendingSum) and getattr(self.final_norm, "takes_pending_sum", False)):
            pending = None                      # a block that adds into the stream itself left it complete
        if h.dim() == 3:
            # the output reads the sum of the streams; a norm without statistics joins that kernel
            from ..kernels import ops
            fused = self.final_norm.elementwise() if hasattr(self.final_norm, "elementwise") else None
            xn = ops.streams_read(h, None, fused, ctx.act_dtype, rows=logit_rows)
            if fused is None:
                xn = self.final_norm.forward(xn, ctx.act_dtype)
        else:
            xn = self.final_norm.gather_forward(h, pending, logit_rows, ctx.act_dtype)
        return self.head.forward(xn)


def _sub(part_spec) -> str:
    """Tensor-name segment between the layer prefix and a part's tensors: the spec's
    ``tensor_prefix`` (none: the part's tensors lie directly under the layer prefix)."""
    sub = part_spec.get().get("tensor_prefix")
    return "" if sub is None else str(sub)
