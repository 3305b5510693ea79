"""Drop-in encode / decode for the reference's residual vector quantisers on B200.

``MimiRVQB200`` mirrors ``MimiResidualVectorQuantizer`` (src/fast_mimi/model.py:2365-2444): ``encode(embeddings
[B, hidden, T], num_quantizers) -> int64 [K, B, T]`` and ``decode(codes [B, K, T]) -> float32 [B, hidden, T]``;
``MimiSplitRVQB200`` mirrors ``MimiSplitResidualVectorQuantizer`` (src/fast_mimi/model.py:2447-2480): one semantic
stack plus one acoustic stack on the same embeddings.  The 1 x 1 convolutions ``input_proj`` / ``output_proj`` run on
the tensor core as split-precision products (``ops.linear_split``: FP16 hi + lo parts, FP32 accumulation, the accuracy
of an FP32 linear, which the code decisions downstream need), the codebook search on ``ops.rvq_encode`` (tensor-core pre-selection, exact FP32 decision) and the
ordered sum on ``ops.rvq_decode``.  Codebook vectors are taken from the reference modules
(``layer.codebook.embed``) when the wrapper is built; rebuild it after loading new weights.
"""
from __future__ import annotations

import torch
import torch.nn as nn

from . import _native, ops


class _Frames:
    """Embeddings ``[B, C, T]`` as frame-major float32 rows; their FP16 hi + lo parts, if asked for, are made once for all branches."""

    def __init__(self, embeddings: torch.Tensor) -> None:
        B, _, T = embeddings.shape
        self.rows = embeddings.float().permute(0, 2, 1).reshape(B * T, -1).contiguous()
        self._parts = None

    def parts(self):
        if self._parts is None:
            self._parts = ops.split_half(self.rows)
        return self._parts


class MimiRVQB200:
    def __init__(self, codebooks: torch.Tensor, input_proj: torch.Tensor | None, output_proj: torch.Tensor | None) -> None:
        self.books = ops.RVQCodebooks(codebooks)
        flat = lambda w: None if w is None else w.detach().float().reshape(w.shape[0], -1).contiguous()
        self.input_proj, self.output_proj = flat(input_proj), flat(output_proj)
        # FP16 hi + lo parts of the projection weights for the tensor-core products
        self._in_parts = None if self.input_proj is None else ops.split_half(self.input_proj)
        self._out_parts = None if self.output_proj is None else ops.split_half(self.output_proj)

    @staticmethod
    def _on_tensor_core(w: torch.Tensor) -> bool:
        # the tensor-core kernel takes K in multiples of 64 and N in multiples of 256 (Mimi: 512 -> 256 and back);
        # other geometries (the reference's tiny test configuration) take the FP32 CUDA-core kernel
        return w.shape[1] % 64 == 0 and w.shape[0] % 256 == 0

    @classmethod
    def from_reference(cls, rvq: nn.Module) -> "MimiRVQB200":
        """``rvq``: a module with the reference's attributes ``layers[i].codebook.embed``, ``input_proj``,
        ``output_proj`` (1 x 1 ``nn.Conv1d`` without bias, or ``None``)."""
        books = torch.stack([layer.codebook.embed.detach().float() for layer in rvq.layers])
        weight = lambda conv: None if conv is None else conv.weight
        return cls(books, weight(rvq.input_proj), weight(rvq.output_proj))

    def encode(self, embeddings: torch.Tensor, num_quantizers: int | None = None) -> torch.Tensor:
        ops._need(embeddings.is_cuda and embeddings.dim() == 3, "embeddings must be CUDA [batch, channels, frames]")
        B, _, T = embeddings.shape
        layers = self._layers(num_quantizers)
        codes = torch.empty(layers, B * T, dtype=torch.int64, device=embeddings.device)
        self._encode_frames(_Frames(embeddings), codes)
        # codes are the end of the device pipeline: a recorded error (a timed-out wait in a kernel upstream, a
        # non-finite residual) must not leave as plausible-looking indices
        ops.check_status(embeddings.device)
        return codes.view(layers, B, T)

    def _layers(self, num_quantizers: int | None) -> int:
        layers = self.books.layers if num_quantizers is None else int(num_quantizers)
        ops._need(0 < layers <= self.books.layers, "num_quantizers out of range")
        return layers

    def _encode_frames(self, frames: "_Frames", codes: torch.Tensor, x: torch.Tensor | None = None) -> None:
        """Codes of the first ``len(codes)`` layers into ``codes [layers, frames]``; nothing is read back.  ``x``: the frames
        after the projection, if they are at hand (overwritten)."""
        if x is not None:
            pass
        elif self.input_proj is None:
            x = frames.rows.clone()
        elif self._on_tensor_core(self.input_proj):
            x = ops._linear_rows(frames.rows, frames.parts, self._in_parts, (len(frames.rows),), None)
        else:
            x = ops.linear_fp32(frames.rows, self.input_proj)
        ops._need(x.shape[1] == ops.RVQ_DIM, "x must be CUDA float32 [rows, 256]")
        ops._rvq_search(x, self.books, codes, None, ops._status_ptr(None, x))

    def decode(self, codes: torch.Tensor) -> torch.Tensor:
        ops._need(codes.is_cuda and codes.dim() == 3, "codes must be CUDA [batch, quantizers, frames]")
        B, K, T = codes.shape
        if self.output_proj is not None and self._on_tensor_core(self.output_proj):
            return ops.rvq_decode_project(codes, self.books, None, self._out_parts)
        q = ops.rvq_decode(codes.transpose(0, 1).reshape(K, B * T).contiguous(), self.books)
        if self.output_proj is not None:
            q = ops.linear_fp32(q, self.output_proj)
        return q.view(B, T, -1).permute(0, 2, 1).contiguous()


class MimiSplitRVQB200:
    _joint_in: tuple | None = None          # of the class, so that quantisers pickled before there were joint projections
    _joint: tuple | None = None             # make theirs on the first call

    def __init__(self, semantic: MimiRVQB200, acoustic: MimiRVQB200) -> None:
        self.semantic, self.acoustic = semantic, acoustic
        self.num_semantic_quantizers = semantic.books.layers
        self.max_num_quantizers = semantic.books.layers + acoustic.books.layers
        self._joint_in_parts()
        self._joint_out_parts()

    def _joint_in_parts(self):
        """Both input projections as one weight ``[2 * 256, hidden]``, so that the embeddings are read once."""
        sem, aco = self.semantic, self.acoustic
        w0, w1 = sem.input_proj, aco.input_proj
        if self._joint_in is None or self._joint_in[0] is not w0 or self._joint_in[1] is not w1:
            fits = (w0 is not None and w1 is not None and w0.shape == w1.shape and w0.shape[0] == ops.RVQ_DIM
                    and sem._on_tensor_core(w0) and w0.device == w1.device)
            self._joint_in = (w0, w1, ops.split_half(torch.cat((w0, w1), dim=0)) if fits else None)
        return self._joint_in[2]

    def _joint_out_parts(self):
        """Both output projections as one weight over [semantic | acoustic], whose product adds the branches; made once for a
        pair of branches, ``None`` where they do not fit together."""
        sem, aco = self.semantic, self.acoustic
        w0, w1 = sem.output_proj, aco.output_proj
        if self._joint is None or self._joint[0] is not w0 or self._joint[1] is not w1:
            fits = w0 is not None and w1 is not None and w0.shape == w1.shape and sem._on_tensor_core(w0) and w0.device == w1.device
            self._joint = (w0, w1, ops.split_half(torch.cat((w0, w1), dim=1)) if fits else None)
        return self._joint[2]

    @classmethod
    def from_reference(cls, split: nn.Module) -> "MimiSplitRVQB200":
        return cls(MimiRVQB200.from_reference(split.semantic_residual_vector_quantizer),
                   MimiRVQB200.from_reference(split.acoustic_residual_vector_quantizer))

    def encode(self, embeddings: torch.Tensor, num_quantizers: int | None = None) -> torch.Tensor:
        count = self.max_num_quantizers if num_quantizers is None else int(num_quantizers)
        if not self.num_semantic_quantizers <= count <= self.max_num_quantizers:
            raise ValueError(f"num_quantizers must be in [{self.num_semantic_quantizers}, {self.max_num_quantizers}]")
        ops._need(embeddings.is_cuda and embeddings.dim() == 3, "embeddings must be CUDA [batch, channels, frames]")
        B, _, T = embeddings.shape
        n_sem = self.semantic._layers(None)
        acoustic = count - self.num_semantic_quantizers
        x = [None, None]
        parts = None
        if acoustic > 0:
            self.acoustic._layers(acoustic)
            parts = self._joint_in_parts()
            if parts is not None:
                sem, aco = self.semantic.books, self.acoustic.books
                made = _native.bind().rvq_encode(embeddings, *parts, (sem._native(n_sem), aco._native(acoustic)), ops.RVQ_TAU_REL[torch.float32],
                                                 ops.default_status(embeddings.device))
                if type(made) is int:
                    ops._raise_status(made)
                if made is not None:
                    return ops._made(made)
        codes = torch.empty(n_sem + acoustic, B * T, dtype=torch.int64, device=embeddings.device)
        frames = _Frames(embeddings)
        if parts is not None:
            x = ops._linear_rows(frames.rows, frames.parts, parts, (B * T,), None, mats=2)
            if self.semantic.books.entries == self.acoustic.books.entries:
                ops._rvq_search_stacks(x, (self.semantic.books, self.acoustic.books), (codes[:n_sem], codes[n_sem:]), ops._status_ptr(None, x))
                ops.check_status(embeddings.device)
                return codes.view(len(codes), B, T)
        self.semantic._encode_frames(frames, codes[:n_sem], x[0])
        if acoustic > 0:
            self.acoustic._encode_frames(frames, codes[n_sem:], x[1])
        ops.check_status(embeddings.device)
        return codes.view(len(codes), B, T)

    def decode(self, codes: torch.Tensor) -> torch.Tensor:
        """``codes [B, K, T]``: semantic layers first (src/fast_mimi/model.py:2408-2444 per branch); the two
        branches' outputs are added."""
        n_sem = self.num_semantic_quantizers
        if codes.is_cuda and codes.dim() == 3 and n_sem == self.semantic.books.layers < codes.shape[1]:
            parts = self._joint_out_parts()
            if parts is not None:
                return ops.rvq_decode_project(codes, self.semantic.books, self.acoustic.books, parts)
        out = self.semantic.decode(codes[:, :n_sem].contiguous())
        if codes.shape[1] > n_sem:
            out = out + self.acoustic.decode(codes[:, n_sem:].contiguous())
        return out
