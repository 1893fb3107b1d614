"""All layers of a decode step issued as one cooperative kernel (`csrc/decode_step.cu`).

A step of few sequences that bring one token each is, launch by launch, a chain of eight dependent kernels a layer, each of
which takes longer than its share of the weights takes to read.  `DecodeStep` hands the whole run of layers to one kernel
whose CTAs live for the step.  It serves pre-norm blocks of the package's own attention (heads of 64 or 128, no window, its own
cache), silu-gated feed-forward and RMS norm parts in bfloat16, all of equal sizes; `DecodeStep.of` says whether a model is
one, `takes` whether a step is.  Every other step keeps the layer-by-layer path.
"""

from __future__ import annotations

import ctypes
import weakref

import torch

from . import build

_c = ctypes
_P, _I, _F, _LL = _c.c_void_p, _c.c_int, _c.c_float, _c.c_longlong


class StepLayer(_c.Structure):
    """ShrikeStepLayer."""

    _fields_ = [(name, _P) for name in ("w_qkv", "w_o", "w_gate_up", "w_down", "norm_mixer", "norm_ffn", "b_qkv", "keys", "values")] + [
        ("eps_mixer", _F), ("eps_ffn", _F)]


class StepArgs(_c.Structure):
    """ShrikeStepArgs."""

    _fields_ = (
        [(name, _P) for name in ("layers", "positions", "slots", "block_table", "ctx_len", "inv_freq", "resid", "words", "sync", "status")]
        + [("num_slots", _LL)]
        + [(name, _I) for name in ("num_layers", "tokens", "width", "heads", "kv_heads", "head_dim", "inter", "max_blocks", "page_size",
                                   "num_pages")]
        + [("scale", _F)]
    )


class DecodeStep:
    MAX_TOKENS = 8
    NOT_TOGETHER = -2   # the launcher's answer where the device will not run all CTAs at once

    def __init__(self, ops, runtime, blocks, order):
        self.ops, self.runtime, self.blocks, self.order = ops, runtime, blocks, order
        self.lib = build.decode_step_library()
        self.lib.shrike_decode_step_keys.argtypes = [_I] * 7
        self.lib.shrike_decode_step_words.argtypes = [_I] * 6
        self.lib.shrike_decode_step_table.argtypes = [_P, _I, _I, _I, _I, _I, _I, _P]
        self.lib.shrike_decode_step.argtypes = [_P, _P]
        for name in ("keys", "table", "layer_bytes"):
            getattr(self.lib, f"shrike_decode_step_{name}").restype = _I
        self.lib.shrike_decode_step_words.restype = _LL
        self.lib.shrike_decode_step.restype = _I
        mixer, ffn = blocks[order[0].layer].mixer.spec, blocks[order[0].layer].feed_forward.spec
        self.sizes = (mixer.width, mixer.num_heads, mixer.num_kv_heads, mixer.head_dim, ffn.intermediate)
        self._storage = None   # weakly: the pool the table's addresses belong to
        self._table = self._words = self._sync = None
        self._most_keys: dict[int, int] = {}   # sequences -> the longest context served
        self._refused = False   # by the device, at a launch

    @classmethod
    def of(cls, ops, runtime, blocks, order):
        """The program for a model of these blocks, or None where they are not what it serves."""
        from ..parts.attention import PagedAttention
        from ..parts.block import PreNormBlock
        from ..parts.mlp import GatedMLP
        from ..parts.norm import RMSNorm

        if not getattr(ops, "whole_steps", False) or not order:
            return None
        sizes, turns = set(), []
        for run in order:
            block = blocks[run.layer]
            if type(block) is not PreNormBlock or run.enter is not None or not run.writes_cache:
                return None
            if (type(block.mixer), type(block.feed_forward)) != (PagedAttention, GatedMLP):
                return None
            if (type(block.mixer_norm), type(block.feed_forward_norm)) != (RMSNorm, RMSNorm):
                return None
            spec, ffn = block.mixer.spec, block.feed_forward.spec
            position = block.mixer.position
            if spec.window is not None or block.mixer.b_o is not None or ffn.activation != "silu" or block.feed_forward.run != 16:
                return None
            table = None if position is None else position.rotary_table()
            if position is not None and table is None:
                return None
            turns.append(table)
            sizes.add((spec.width, spec.num_heads, spec.num_kv_heads, spec.head_dim, spec.scale, ffn.intermediate))
        if len(sizes) != 1 or len({run.cache for run in order}) != len(order):
            return None
        first = turns[0]   # one rotation for all layers
        if any((t is None) != (first is None) or (t is not None and t is not first and not torch.equal(t, first)) for t in turns):
            return None
        program = cls(ops, runtime, blocks, order)
        return program if program.most_keys(1) > 0 else None

    def most_keys(self, tokens: int) -> int:
        """The longest context of a step of `tokens` sequences that is served (0: none)."""
        held = self._most_keys.get(tokens)
        if held is None:
            held = self._most_keys[tokens] = self.lib.shrike_decode_step_keys(tokens, len(self.order), *self.sizes)
        return held

    def takes(self, step) -> bool:
        """Whether a step is run here; `step` is a `StepContext`, or a `Staged` step whose captured form is looked for."""
        # keys of earlier positions are read while this step's are still being written: no entry may bring another's
        return (not self._refused and step.all_single and step.apart and step.num_tokens <= self.MAX_TOKENS
                and getattr(self.ops, "whole_steps", False) and step.max_ctx_len <= self.most_keys(step.num_tokens))

    def _tables(self, storage) -> None:
        """The layers' addresses on the device, written once per cache pool."""
        if self._storage is not None and self._storage() is storage:
            return
        width, heads, kv_heads, dim, inter = self.sizes
        layers = (StepLayer * len(self.order))()
        for entry, run in zip(layers, self.order):
            block = self.blocks[run.layer]
            mixer, ffn = block.mixer, block.feed_forward
            _group, keys, values = storage.keys_values(run.cache)
            entry.w_qkv, entry.w_o = mixer.w_qkv.data_ptr(), mixer.w_o.data_ptr()
            entry.w_gate_up, entry.w_down = ffn.w_gate_up.data_ptr(), ffn.w_down.data_ptr()
            entry.norm_mixer, entry.norm_ffn = block.mixer_norm.weight.data_ptr(), block.feed_forward_norm.weight.data_ptr()
            entry.b_qkv = None if mixer.b_qkv is None else mixer.b_qkv.data_ptr()
            entry.keys, entry.values = keys.data_ptr(), values.data_ptr()
            entry.eps_mixer, entry.eps_ffn = block.mixer_norm.spec.eps, block.feed_forward_norm.spec.eps
        host = torch.empty(len(self.order) * self.lib.shrike_decode_step_layer_bytes(), dtype=torch.uint8)
        with torch.cuda.device(self.ops.device):
            rc = self.lib.shrike_decode_step_table(layers, len(self.order), width, heads, kv_heads, dim, inter, host.data_ptr())
        self._check(rc)
        device = self.ops.device
        self._table = host.to(device)
        if self._words is None:
            count = self.lib.shrike_decode_step_words(self.MAX_TOKENS, *self.sizes)
            self._words = torch.zeros(count, dtype=torch.int64, device=device)
            self._sync = torch.tensor([1, 0], dtype=torch.int32, device=device)
        self._storage = weakref.ref(storage)
        self.ops.generation += 1

    @staticmethod
    def _check(rc: int) -> None:
        if rc != 0:
            from .cuda_ops import KernelError

            raise KernelError(f"decode_step: launcher returned {rc}")

    def run(self, resid, ctx):
        """Runs the layers on `resid` [N, W] float32, in place: nothing is left pending.  False where the device will not run the
        kernel's CTAs together: nothing has run then, and no step is taken any more."""
        self._tables(ctx.storage)
        width, heads, kv_heads, dim, inter = self.sizes
        mixer = self.blocks[self.order[0].layer].mixer
        group, keys, _values = ctx.storage.keys_values(self.order[0].cache)
        view = ctx.groups[group]
        table = mixer.position.rotary_table() if mixer.position is not None else None
        args = StepArgs(
            layers=self._table.data_ptr(), positions=ctx.positions.data_ptr(), slots=view.slot_mapping.data_ptr(),
            block_table=view.block_table.data_ptr(), ctx_len=ctx.ctx_len.data_ptr(),
            inv_freq=None if table is None else table.data_ptr(), resid=resid.data_ptr(), words=self._words.data_ptr(),
            sync=self._sync.data_ptr(), status=self.ops.status.data_ptr(), num_slots=keys.shape[0] * keys.shape[1],
            num_layers=len(self.order), tokens=ctx.num_tokens, width=width, heads=heads, kv_heads=kv_heads, head_dim=dim, inter=inter,
            max_blocks=view.max_blocks, page_size=keys.shape[1], num_pages=keys.shape[0], scale=mixer.spec.scale)
        rc = self.lib.shrike_decode_step(_c.byref(args), self.ops._stream())
        self._refused = rc == self.NOT_TOGETHER
        if self._refused:
            return False
        self._check(rc)
        self.ops.launches += 1
        return True
