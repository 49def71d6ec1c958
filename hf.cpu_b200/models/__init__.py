"""A model put together from a plan: parts per layer, the run order, weights bound by name.

``Model.forward`` is the forward pass the step function drives: embedding, the schedule's
entries in order, then the final norm and the head on the rows whose logits are wanted
(src/model.c:545-640).
"""
from __future__ import annotations

import operator
import os
from dataclasses import dataclass
from functools import lru_cache
from typing import Dict, List, Optional

import torch

from .. import kernels
from ..config import ModelConfig, load_config
from ..config.base import ModelPlan
from ..parts import Part, make_part
from ..weights import RandomSource, TensorSpec, load_tensors


EMBEDDING_STATE = "embedding"        # the key of the embedding's per-request state among the schedule entries' states


def block_state_key(entry: int):
    """The key of a block's own per-request state (a token shift's previous row) for schedule entry ``entry``; a layer
    that runs more than once has one per run."""
    return ("block", entry)


@dataclass
class Layer:
    block: object
    norm1: object
    mixer: object
    norm2: object
    ffn: object
    post1: object = None
    post2: object = None
    changes = 0                  # (no field: how many times one has been set)

    def __setattr__(self, name, value):
        super().__setattr__(name, value)
        vars(self)["changes"] = self.changes + 1

    def parts(self):
        return tuple(p for p in (self.block, self.norm1, self.mixer, self.post1, self.norm2, self.ffn, self.post2)
                     if p is not None)

    def post_norms(self):
        """Keyword arguments for the block, for arrangements with norms behind the sublayers."""
        return {"post1": self.post1, "post2": self.post2} if self.post1 is not None else {}


@lru_cache(maxsize=64)
def _written(*classes) -> kernels.Written:
    """The functions of parts' classes as they were written (kept here and not by the models, which can be copied and stored)."""
    return kernels.Written.together(c.written for c in classes)


class Model:
    _alike = _watched = ()            # what is found when the weights are bound

    def __init__(self, config: ModelConfig, run_dtype: torch.dtype = torch.bfloat16,
                 device: torch.device = torch.device("cuda:0"), plan: Optional[ModelPlan] = None):
        if run_dtype not in (torch.bfloat16, torch.float32):
            raise ValueError(f"run dtype must be bfloat16 or float32, got {run_dtype}")
        self.config, self.run_dtype, self.device = config, run_dtype, torch.device(device)
        self.plan = plan if plan is not None else config.plan()
        self.plan.validate()
        p = self.plan
        self.positions = {name: make_part("position", spec) for name, spec in p.positions.items()}
        self.embedding = make_part("embedding", p.embedding)
        self.transitions = {name: make_part("transition", spec) for name, spec in p.transitions.items()}
        self.layers: List[Layer] = []
        for ls in p.layers:
            self.layers.append(Layer(
                block=make_part("block", ls.block),
                norm1=make_part("norm", ls.norm1),
                mixer=make_part("mixer", ls.mixer, positions=self.positions),
                norm2=make_part("norm", ls.norm2) if ls.norm2 is not None else None,
                ffn=make_part("ffn", ls.ffn) if ls.ffn is not None else None,
                post1=make_part("norm", ls.post_norm1) if ls.post_norm1 is not None else None,
                post2=make_part("norm", ls.post_norm2) if ls.post_norm2 is not None else None))
        self.final_norm = make_part("norm", p.final_norm)
        self.head = make_part("head", p.head)
        self.bound = False
        self.files: List[str] = []            # the weight files this model was loaded from

    # ---- weights ------------------------------------------------------------------------
    def all_parts(self):
        yield self.embedding
        yield from self.positions.values()
        yield from self.transitions.values()
        for l in self.layers:
            yield from l.parts()
        yield self.final_norm
        yield self.head

    def tensor_specs(self) -> List[TensorSpec]:
        seen: Dict[str, TensorSpec] = {}
        for part in self.all_parts():
            for s in part.tensor_specs():
                if s.name in seen and seen[s.name].shape != s.shape:
                    raise ValueError(f"tensor '{s.name}' is declared with two shapes")
                seen.setdefault(s.name, s)
        return list(seen.values())

    def bind(self, tensors) -> "Model":
        """Hand the weights to the parts.  ``tensors`` maps names to tensors: a dict, or a source that makes
        each tensor when it is asked for, so that the parts take them one at a time."""
        if hasattr(tensors, "keep"):
            # a tensor that two parts bind (a tied head reads the embedding) is made once
            count: Dict[str, int] = {}
            for part in self.all_parts():
                for s in part.tensor_specs():
                    count[s.name] = count.get(s.name, 0) + 1
            tensors.keep(n for n, c in count.items() if c > 1)
        for part in self.all_parts():
            part.bind(tensors, self.run_dtype, self.device)
        for l in self.layers:
            l.block.join_outputs(l.mixer, l.ffn)
        for pos in self.positions.values():
            pos.prepare(self.plan.max_positions, self.device)
        self._look_for_alike()
        self.bound = True
        return self

    def _replay_parts(self, i: int):
        """The parts whose kernels schedule entry ``i`` runs: its layer's, and the norm its block may write for the next."""
        l = self.layers[self.plan.schedule[i].layer]
        return l.norm1, l.mixer, l.norm2, l.ffn, self.layers[self.plan.schedule[i + 1].layer].norm1

    def _replay_tensors(self, i: int, cache):
        a, b, c, d, e = self._replay_parts(i)
        own = (*a.replay_tensors(), *b.replay_tensors(), *c.replay_tensors(), *d.replay_tensors(), *e.replay_tensors())
        return own if cache is None else (*own, cache.k, cache.v)

    def _look_for_alike(self) -> None:
        """``_alike``: for each schedule entry a number that entries share whose kernels differ in their tensors only; None for the
        last entry and those with a part, a state or a step in front that says otherwise."""
        numbers, self._alike, watched, schedule = {}, [], [], self.plan.schedule
        for i, e in enumerate(schedule):
            key = None
            if i + 1 < len(schedule):
                l, following = self.layers[e.layer], schedule[i + 1]
                after = self.layers[following.layer]
                if (e.enter is None and following.enter is None and e.cache_of is None and l.ffn is not None and l.norm2 is not None
                        and not l.post_norms() and l.mixer.state_spec() is None and l.block.state_spec() is None):
                    parts = (l.block, after.block) + self._replay_parts(i)
                    keys = tuple(p.replay_key() if isinstance(p, Part) and p.counts_changes and p.written.names.isdisjoint(vars(p)) else None for p in parts)
                    if all(k is not None for k in keys):
                        key = keys
                        watched += [l, after, *parts]
            self._alike.append(None if key is None else numbers.setdefault(key, len(numbers)))
        # layers and parts as they were, and the functions of their classes
        self._watched = list({id(o): o for o in watched}.values())
        self._changes_then, self._layers_then = [o.changes for o in self._watched], list(self.layers)
        self._classes = tuple(dict.fromkeys(type(o) for o in self._watched if isinstance(o, Part)))

    def _alike_now(self) -> Optional[List[Optional[int]]]:
        """``_alike``, None where no entries are.  What has been changed since the weights were bound (an attribute of a part, a
        function put over one of its own, another part in its place) is alike with nothing: its own code runs."""
        if not self._watched or not _written(*self._classes).holds():
            return None
        if [o.changes for o in self._watched] == self._changes_then and len(self.layers) == len(self._layers_then) and \
                all(map(operator.is_, self.layers, self._layers_then)):
            return self._alike
        same = {id(o) for o, n in zip(self._watched, self._changes_then) if o.changes == n}
        out = []
        for i, number in enumerate(self._alike):
            if number is not None:
                l, after = self.layers[self.plan.schedule[i].layer], self.layers[self.plan.schedule[i + 1].layer]
                if not all(id(o) in same for o in (l, after, l.block, after.block) + self._replay_parts(i)):
                    number = None
            out.append(number)
        return out

    def weight_bytes_per_step(self) -> int:
        """Bytes of weights one decode step reads: every schedule entry's layer and the head, once each."""
        total = self.head.weight_bytes() + self.final_norm.weight_bytes()
        for e in self.plan.schedule:
            total += sum(p.weight_bytes() for p in self.layers[e.layer].parts())
            if e.enter is not None:
                total += self.transitions[e.enter[0]].weight_bytes()
        return total

    # ---- forward ------------------------------------------------------------------------
    def forward(self, ctx) -> Optional[torch.Tensor]:
        T = ctx.token_ids.shape[0]
        S = self.plan.streams
        x = ctx.buf("residual", (T, self.plan.hidden_size), torch.float32)
        self.embedding.forward(ctx.token_ids, x, ctx=ctx, state=ctx.entry_state(EMBEDDING_STATE))
        if S > 1:
            # the stream in S copies, a token's copies side by side, all equal to the embedding at the start
            emb, x = x, ctx.buf("residual_copies", (T, S * self.plan.hidden_size), torch.float32)
            with kernels.phase("glue"):
                kernels.hc_spread(emb, x, S)
        schedule = self.plan.schedule
        for tr in self.transitions.values():
            tr.begin(ctx, x)
        xn = None                                # norm1 of the coming block, when the previous block computed it
        record = kernels.recorder() if self._watched else None
        alikes = self._alike_now() if record is not None else None
        model = None                             # ((number, input, cache group), launches, output) of a layer that was written down
        for i, e in enumerate(schedule):
            layer = self.layers[e.layer]
            owner = i if e.cache_of is None else e.cache_of
            alike = alikes[i] if alikes is not None else None
            if alike is not None:
                cache = ctx.entry_cache(i)
                like = alike, None if xn is None else xn.data_ptr(), None if cache is None else cache.group
                if model is not None and model[0] == like and model[1].replay(self._replay_tensors(i, cache)):
                    xn = model[2]
                    continue
                if alikes[i + 1] != alike or (model is not None and model[0] == like):
                    alike = None                 # (no layer that would make the same calls follows)
            # the norm that follows this block: the next block's first, or, after the last block of a step whose
            # tokens all want their logits (a step of single tokens), the final norm
            extra = layer.post_norms()
            if e.enter is not None:
                # (what the block in front handed over is the transition's operand; the layer's input comes out of it)
                out = ctx.buf("enter_xn", x.shape, self.run_dtype) if layer.block.state_spec() is None else None
                done = self.transitions[e.enter[0]].enter(ctx, x, e.enter[1], xn, layer.norm1 if out is not None else None, out)
                xn = out if done else None
            if i + 1 < len(schedule) and schedule[i + 1].enter is not None:
                next_norm = self.transitions[schedule[i + 1].enter[0]].operand_norm()
                if getattr(layer.block, "wants_next_block", False):
                    extra["next_block"] = None
            elif i + 1 < len(schedule):
                next_norm = self.layers[schedule[i + 1].layer].norm1
                following = self.layers[schedule[i + 1].layer].block
                if getattr(layer.block, "wants_next_block", False):
                    extra["next_block"] = following
                if following.state_spec() is not None:
                    # a block with state of its own (a token shift) makes its mixer's input itself, unless the block in
                    # front knows how to
                    if getattr(layer.block, "fuses_next_shift", False):
                        extra["next_block_state"] = ctx.entry_state(block_state_key(i + 1))
                    else:
                        next_norm = None
            else:
                next_norm = self.final_norm if getattr(ctx, "logits_for_all", False) else None
            if layer.block.state_spec() is not None:
                extra["block_state"] = ctx.entry_state(block_state_key(i))

            def run():
                return layer.block.forward(ctx, x, layer.norm1, layer.mixer, layer.norm2, layer.ffn,
                                           ctx.entry_cache(owner), ctx.entry_state(i), e.cache_of is None,
                                           xn_ready=xn, next_norm=next_norm, **extra)
            if alike is None:
                xn = run()
            else:
                xn, calls = record(run, self._replay_tensors(i, cache))
                model = (like, calls, xn) if calls is not None else None
        M = ctx.num_logit_rows
        if M == 0:
            return None
        if xn is None or not schedule:
            xn = ctx.buf("head_xn", (M, self.plan.hidden_size), self.run_dtype)
            if S > 1:
                # the head reads the sum of the copies
                params = getattr(self.final_norm, "params", None)
                with kernels.phase("glue"):
                    if params is not None:
                        kernels.hc_in_norm(x, S, None, ctx.logit_rows, params, xn)
                    else:
                        total = ctx.buf("head_sum", (M, self.plan.hidden_size), torch.float32)
                        kernels.hc_in_norm(x, S, None, ctx.logit_rows, None, total)
                        self.final_norm.forward(total, xn)
            else:
                self.final_norm.forward(x, xn, rows=ctx.logit_rows)
        logits = ctx.buf("logits", (M, self.plan.vocab_size), torch.float32)
        self.head.forward(xn, logits)
        return logits


def build_model_specs(config: ModelConfig) -> List[TensorSpec]:
    return Model(config, torch.float32, torch.device("cpu")).tensor_specs()


def load_model(path: str, dtype: torch.dtype = torch.bfloat16, device="cuda:0") -> Model:
    """Load a model folder (``config.json`` + safetensors: one file, or shards with or without an index) or one of
    the reference's GGUF files; the model class follows the configuration.  Every tensor is checked against the
    model's declaration before any is read, and tensors go to the device one at a time."""
    if os.path.isfile(path) and path.endswith(".gguf"):
        return load_gguf_model(path, dtype, device)
    config = load_config(path)
    model = Model(config, dtype, torch.device(device))
    tensors = load_tensors(path, model.tensor_specs(), dtype, model.device)
    try:
        model.bind(tensors)
        model.files = tensors.paths()
    finally:
        tensors.close()
    return model


def load_gguf_model(path: str, dtype: torch.dtype = torch.bfloat16, device="cuda:0") -> Model:
    """The same from one of the reference's own GGUF files (float tensor types only)."""
    from ..weights.gguf import GgufSource
    tensors = GgufSource(path, dtype, torch.device(device))
    try:
        model = Model(tensors.config, dtype, torch.device(device))
        tensors.check(model.tensor_specs())
        model.bind(tensors)
        model.files = [path]
    finally:
        tensors.close()
    return model


def random_model(config: ModelConfig, seed: int = 0, dtype: torch.dtype = torch.bfloat16, device="cuda:0",
                 std: float = 0.02) -> Model:
    """A model with random weights made directly on ``device`` (no files), one tensor at a time."""
    model = Model(config, dtype, torch.device(device))
    store = torch.float32 if dtype == torch.float32 else torch.bfloat16
    return model.bind(RandomSource(model.tensor_specs(), seed, store, model.device, std=std))
