"""A decoder assembled from a :class:`ModelSpec`: embedding, the scheduled runs of its layers, the
final norm and the output head at the wanted rows.

The model is the same object whatever the architecture; which parts it holds and in which order
they run comes from the spec (reference: ``embed`` → every ``layer`` → ``logits`` on the last row,
crates/mrun-engine/src/nuvec_engine.rs:999-1028, crates/mrun-engine/src/models/common.rs:382-414).
"""
from __future__ import annotations

from typing import Dict, List, Optional

import torch

from ..config.spec import ModelSpec
from ..kernels import ops
from ..parts import ARRANGEMENTS, EMBEDDINGS, NORMS, TRANSFORMS, Runtime
from ..parts.base import local
from .batch import StepContext


class Model:
    def __init__(self, spec: ModelSpec, tensors: Dict[str, torch.Tensor], runtime: Runtime):
        spec.validate()
        if spec.streams < 1 or (spec.streams > 1 and spec.embedding_transform is not None):
            raise ValueError("a model has at least one residual stream; an embedding transform takes one stream")
        self.spec = spec
        self.runtime = runtime
        self.embedding = runtime.matrix(tensors[spec.embedding_name])
        if self.embedding.shape != (spec.vocab_size, spec.hidden_size):
            raise ValueError("the embedding table does not have the spec's shape")
        # an embedding part in place of the plain lookup: it gets the token table (as the model
        # holds it) under the empty name and its other tensors by their own names
        self.embedder = None
        if spec.embedding is not None:
            if spec.tie_embeddings:
                raise ValueError("an embedding part does not share its table with the output head")
            mine = {t.name: tensors[t.name] for t in EMBEDDINGS.tensor_specs(spec.embedding, spec.embedding_name)
                    if t.name in tensors and t.name != spec.embedding_name}
            mine[""] = self.embedding
            self.embedder = EMBEDDINGS.build(spec.embedding, mine, runtime)
        self.head = self.embedding if spec.tie_embeddings else runtime.matrix(tensors[spec.head_name])
        self.blocks = [ARRANGEMENTS.get(layer.arrangement)(layer, tensors, runtime) for layer in spec.layers]
        self.final_norm = NORMS.build(spec.final_norm, local(tensors, spec.final_norm_prefix), runtime)
        self.order = spec.run_order()
        self.embedding_transform = self.logits_transform = None
        if spec.embedding_transform is not None:
            t = spec.embedding_transform
            self.embedding_transform = TRANSFORMS.build(t, local(tensors, getattr(t, "prefix", "")), runtime)
        if spec.logits_transform is not None:
            t = spec.logits_transform
            self.logits_transform = TRANSFORMS.build(t, local(tensors, getattr(t, "prefix", "")), runtime)

    # ------------------------------------------------------------------ cache layout
    def cache_needs(self) -> List[object]:
        """The need of each schedule entry (None for entries that read another's cache)."""
        needs = []
        for entry in self.order:
            block = self.blocks[entry.layer]
            # a block that keeps state of its own (an input convolution) states the need itself
            owner = block if hasattr(block, "cache_need") else block.mixer
            needs.append(None if entry.cache_of is not None else owner.cache_need())
        if self.embedder is not None:       # the embedding part's state comes after the schedule's entries
            needs.append(self.embedder.cache_need())
        return needs

    def cache_shares(self) -> List[Optional[int]]:
        return [entry.cache_of for entry in self.order] + ([None] if self.embedder is not None else [])

    def activation_elements(self) -> int:
        """The widest set of per-token temporaries any part declares (parts without the hint
        count as nothing); the memory budget sizes the step's scratch from it."""
        widest = 0
        for block in self.blocks:
            for part in (getattr(block, "mixer", None), getattr(block, "feed_forward", None)):
                hint = getattr(part, "activation_elements", None)
                if hint is not None:
                    widest = max(widest, int(hint()))
        return widest

    @property
    def graph_safe(self) -> bool:
        return (all(getattr(block.mixer, "graph_safe", False) for block in self.blocks)
                and (self.embedder is None or getattr(self.embedder, "graph_safe", False)))

    def _tensors(self):
        """Every tensor that a part holds, views of one another included."""
        def walk(obj):
            if isinstance(obj, torch.Tensor):
                yield obj
            elif hasattr(obj, "__dict__"):
                for value in vars(obj).values():
                    if isinstance(value, (torch.Tensor,)) or hasattr(value, "__dict__"):
                        yield from walk(value)
                    elif isinstance(value, (list, tuple)):
                        for item in value:
                            yield from walk(item)
        yield from walk(self.final_norm)
        for block in self.blocks:
            yield from walk(block)
        for t in (self.embedding, self.head):
            yield from walk(t)
        if self.embedder is not None:
            yield from walk(self.embedder)

    def weight_bytes(self) -> int:
        storages = (t.untyped_storage() for t in self._tensors())      # views of one tensor share it and count once
        return sum({storage.data_ptr(): storage.nbytes() for storage in storages}.values())

    def product_scratch(self, tokens: int) -> int:
        """Bytes that the largest product of a step of ``tokens`` takes beside its operands and its result."""
        return max((ops.product_scratch(t, tokens) for t in self._tensors()), default=0)

    # ------------------------------------------------------------------ forward
    def hidden_states(self, ctx: StepContext, caches) -> tuple:
        """Runs the layers; returns the 32-bit stream and the last branch output not yet added."""
        ops.RowSums.begin_step(self.runtime.device)
        resid = torch.empty((ctx.num_tokens, self.spec.streams * self.spec.hidden_size), dtype=torch.float32,
                            device=self.runtime.device)
        if self.embedder is not None:
            self.embedder.forward(ctx, caches[len(self.order)], resid, self.spec.streams)
        elif self.spec.streams > 1:         # every stream starts as the embedding's row
            ops.embed_streams(self.embedding, ctx.token_ids, resid, self.spec.streams)
        else:
            ops.embed(self.embedding, ctx.token_ids, resid)
        if self.embedding_transform is not None:
            resid = self.embedding_transform.forward(resid)
        delta = None
        for at, entry in enumerate(self.order):
            block = self.blocks[entry.layer]
            if isinstance(delta, ops.PENDING) and not getattr(block, "accepts_pending", False):
                delta = delta.compute()
            delta = block.forward(resid, delta, ctx, caches[at])
        return resid, delta

    def logits(self, resid: torch.Tensor, delta: Optional[torch.Tensor], rows: torch.Tensor) -> torch.Tensor:
        """float32 ``[len(rows), vocab]``: final norm and head at the wanted rows only."""
        if isinstance(delta, ops.PendingStreams) or self.spec.streams > 1:
            # the last sublayer's write and the sum of the streams, at the wanted rows only
            total = ops.streams_step(resid, delta, None, None, 0.0, torch.float32, self.spec.streams, rows=rows,
                                     want_sum=True)
            h = self.final_norm.add_forward(total, None)
        else:
            if isinstance(delta, ops.PENDING) and not getattr(self.final_norm, "accepts_pending", False):
                delta = delta.compute()
            h = self.final_norm.rows_forward(resid, delta, rows)
        logits = ops.linear(h, self.head, out_dtype=torch.float32)
        if self.logits_transform is not None:
            logits = self.logits_transform.forward(logits)
        return logits

    def forward(self, ctx: StepContext, caches, rows: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
        resid, delta = self.hidden_states(ctx, caches)
        if rows is None or rows.numel() == 0:
            return None
        return self.logits(resid, delta, rows)
