"""Token embedding (pyre/model.py:162,196) and the output head (pyre/model.py:172,201)."""

from __future__ import annotations

import torch

from ..kernels import lib, ops
from ..weights.specs import TensorSpec
from .base import Part, PartSpec, make_part, register_part


class TokenEmbedding(Part):
    """x[t] = table[token[t]], widened to the fp32 residual stream, times ``scale`` (in fp32).  ``norm``: a norm part
    applied to the rows right away (it must offer ``normalize_stream``); its tensors lie under ``norm_prefix`` after
    the table's name."""

    graph_safe = True

    def __init__(self, dtype, device, vocab: int, width: int, tensor_name: str = "weight", norm: "PartSpec | None" = None,
                 norm_prefix: str = ".norm", scale: float = 1.0):
        super().__init__(dtype, device)
        self.vocab, self.width, self.tensor_name = int(vocab), int(width), str(tensor_name)
        self.scale = float(scale)
        self.table = None
        self.norm = make_part("norm", norm, dtype, device) if norm is not None else None
        self.norm_prefix = str(norm_prefix)
        if self.norm is not None and not hasattr(self.norm, "normalize_stream"):
            raise ValueError(f"{type(self.norm).__name__} cannot follow the embedding: it has no normalize_stream")

    def children(self):
        return {self.tensor_name + self.norm_prefix: self.norm} if self.norm is not None else {}

    def tensors(self):
        return {self.tensor_name: TensorSpec((self.vocab, self.width))}

    def load(self, tensors):
        self.table = tensors[self.tensor_name]

    def kernel_libraries(self):
        return ["elementwise"] + (["seqmix"] if self.scale != 1.0 else [])

    def forward(self, ctx):
        x = ops.embedding(self.table, ctx.token_ids, err_flag=ctx.error_flag)
        if self.scale != 1.0:
            ops.scale_cap(x, self.scale)
        return x if self.norm is None else self.norm.normalize_stream(ctx, x)


class LinearHead(Part):
    """fp32 logits = h W^T for the rows that were asked for.  ``tied_to`` names the
    tensor (full checkpoint name) that stands in when the head's own weight is absent:
    the embedding table of a model with tied embeddings (pyre/loader.py:58-61); the
    storage is then shared, not copied.  ``logit_scale``: a factor on the logits; ``softcap`` c > 0: the scaled
    logits become c tanh(logits / c)."""

    graph_safe = True

    def __init__(self, dtype, device, vocab: int, width: int, tied_to: "str | None" = None, tensor_name: str = "weight",
                 logit_scale: float = 1.0, softcap: float = 0.0):
        super().__init__(dtype, device)
        self.vocab, self.width, self.tied_to, self.tensor_name = int(vocab), int(width), tied_to, str(tensor_name)
        self.logit_scale, self.softcap = float(logit_scale), float(softcap)
        self.weight = None

    def tensors(self):
        return {self.tensor_name: TensorSpec((self.vocab, self.width), optional_alias=self.tied_to)}

    def load(self, tensors):
        self.weight = ops.linear_weight(tensors[self.tensor_name])

    def kernel_libraries(self):
        return ops.product_libraries(self.dtype) + (["seqmix"] if self._shaped() else [])

    def _shaped(self) -> bool:
        return self.logit_scale != 1.0 or self.softcap > 0.0

    def forward(self, ctx, h_rows):
        with lib.section("head"):
            logits = ops.linear(h_rows, self.weight, out_dtype=torch.float32)
        return ops.scale_cap(logits, self.logit_scale, self.softcap) if self._shaped() else logits


class NormHeadTail(Part):
    """What follows the last block in this architecture (pyre/model.py:199-201): the final norm, applied to the rows
    whose logits are wanted only (the last block's branch output still pending is added on the way), then the head.
    ``names``: the checkpoint prefixes of the two sub-parts' tensors.  An architecture that ends otherwise (no norm,
    a scaled head, several heads) brings a tail of its own; the model's skeleton is embed, the scheduled blocks, tail."""

    graph_safe = True

    DEFAULT_NAMES = {"norm": "model.norm.", "head": "lm_head."}

    def __init__(self, dtype, device, norm: PartSpec, head: PartSpec, names: "dict[str, str] | None" = None):
        super().__init__(dtype, device)
        self.names = dict(self.DEFAULT_NAMES, **(names or {}))
        self.norm = make_part("norm", norm, dtype, device)
        self.head = make_part("head", head, dtype, device)

    def children(self):
        return {self.names["norm"]: self.norm, self.names["head"]: self.head}

    def forward(self, ctx, x, pending):
        h = self.norm.forward(ctx, x, delta=pending, rows=ctx.logit_rows)
        return self.head.forward(ctx, h)


register_part("embed", "token_embedding", TokenEmbedding)
register_part("tail", "norm_head", NormHeadTail)
register_part("head", "linear_head", LinearHead)
