"""Llama-3 / Qwen2 decoder with the tree hooks of the reference's ``mlx_llama.py``.

``Model(inputs, cache, mask, position_ids, flat_rope)`` keeps the reference's call
(``mlx_llama.py:298-313``): explicit additive mask, integer or per-token array
positions, ``flat_rope`` giving every token of the call the same position.  All
linear layers are 4-bit / group-64 quantised and run through ``libb200eagle.so``;
q/k/v are stored as one fused matrix.  Once the weights are in the streaming layout
(``Model.relayout``) a whole pass is one native call (``b200_forward``: a chain of five kernels per layer, or one
persistent kernel for a tensor-parallel shard); before that, or
with ``model.fused = False``, one layer is nine kernel launches:

    rms_norm -> qmm(+bias) -> rope_kv_append -> tree_attention (+ merge) -> qmm(+residual)
    -> rms_norm -> qmm(SiLU(gate)*up) -> qmm(+residual)

The decode loop does not go through ``__call__`` but through ``forward_device``,
whose inputs (tokens, positions, tail masks, committed length) are read from
device memory, so that a whole speculative step can be replayed as a CUDA graph.
"""
from __future__ import annotations

import collections
import ctypes
import math
import os
from dataclasses import dataclass
from typing import Dict, List, Optional, Union

import torch

from . import _lib
from . import qmm_kernel as qk
from .quantize import quantize

MAX_ROWS = 32          # tokens per forward pass (tree size + 1 <= 32)
MAX_TAIL = 64          # uncommitted cache rows a query can address through its bit mask
MAX_REQUESTS = 4       # requests that can share one forward pass
PREFILL_ROWS = 1024    # prompt tokens per pass of b200_prefill


@dataclass
class ModelArgs:
    """Same fields as ``mlx_llama.py:21-38``."""
    model_type: str
    hidden_size: int
    num_hidden_layers: int
    intermediate_size: int
    num_attention_heads: int
    rms_norm_eps: float
    vocab_size: int
    head_dim: Optional[int] = None
    max_position_embeddings: Optional[int] = None
    num_key_value_heads: Optional[int] = None
    attention_bias: bool = False
    mlp_bias: bool = False
    rope_theta: float = 10000
    rope_traditional: bool = False
    rope_scaling: Optional[Dict[str, Union[float, str]]] = None
    tie_word_embeddings: bool = True

    def __post_init__(self):
        if self.num_key_value_heads is None:
            self.num_key_value_heads = self.num_attention_heads
        if self.head_dim is None:
            self.head_dim = self.hidden_size // self.num_attention_heads
        if self.model_type == "qwen2":
            self.attention_bias = True          # mlx_utils.py:116-117
        if self.rope_traditional:
            raise ValueError("only the non-traditional (half-split) RoPE layout is implemented")
        if self.rope_scaling:
            rope_type = self.rope_scaling.get("type") or self.rope_scaling.get("rope_type")
            if rope_type not in ("linear", "llama3", "default"):
                raise ValueError("rope_scaling type must be linear, llama3 or default")


def rope_inv_freqs(args: ModelArgs):
    """``(inv_freqs fp32 [hd/2], scaling_factor)`` as ``mlx_llama.py:98-116`` builds them."""
    hd = args.head_dim
    idx = torch.arange(0, hd, 2, dtype=torch.float32)
    rope_type = "default"
    if args.rope_scaling:
        rope_type = args.rope_scaling.get("type") or args.rope_scaling.get("rope_type", "default")
    if rope_type in ("default", "linear"):
        scaling = 1.0 / float(args.rope_scaling["factor"]) if rope_type == "linear" else 1.0
        inv = torch.pow(torch.tensor(2.0, dtype=torch.float32), -math.log2(args.rope_theta) * idx / hd)
        return inv.float(), scaling
    # llama3: frequency-dependent rescaling of the base frequencies (mlx_lm rope_utils, Llama3RoPE)
    rs = args.rope_scaling
    factor = float(rs["factor"])
    low = float(rs.get("low_freq_factor", 1.0))
    high = float(rs.get("high_freq_factor", 4.0))
    old_len = float(rs.get("original_max_position_embeddings", 8192))
    freqs = args.rope_theta ** (idx / hd)
    wavelens = 2 * math.pi * freqs
    low_wl, high_wl = old_len / low, old_len / high
    scaled = torch.where(wavelens > low_wl, freqs * factor, freqs)
    smooth = (old_len / wavelens - low) / (high - low)
    mid = freqs / ((1 - smooth) / factor + smooth)
    freqs = torch.where((wavelens > high_wl) & (wavelens < low_wl), mid, scaled)
    return (1.0 / freqs).float(), 1.0


class TensorParallel:
    """Which shard of a tensor-parallel model this process holds (``rank`` of ``world`` GPUs of one node) and
    the ``torch.distributed`` group its all-reduces run in.  q/k/v, gate and up are column-parallel (heads,
    MLP rows), o_proj and down_proj row-parallel (their K is cut; the fp32 partial products are all-reduced
    before the residual add), the vocabulary projection is cut by vocabulary rows."""

    def __init__(self, rank: int, world: int, group=None):
        self.rank, self.world, self.group = int(rank), int(world), group
        # Exchange buffers of the in-kernel all-reduce and argmax combine: one per GPU, mapped into every
        # process of the group through CUDA IPC (addresses as seen by this process, by rank).
        self.peers, self.peer_array = None, None

    def all_reduce_sum(self, t: torch.Tensor):
        import torch.distributed as dist
        dist.all_reduce(t, op=dist.ReduceOp.SUM, group=self.group)

    def all_reduce_max(self, t: torch.Tensor):
        import torch.distributed as dist
        dist.all_reduce(t, op=dist.ReduceOp.MAX, group=self.group)

    def open_exchange(self, hidden: int):
        """Allocate this GPU's exchange buffer, trade IPC handles over the process group and map the
        peers' buffers; returns when every rank has done so (collective call)."""
        import torch.distributed as dist
        lib = _lib.lib()
        nbytes = lib.b200_forward_tp_buffer_bytes(hidden)
        mine, handle = ctypes.c_void_p(), ctypes.create_string_buffer(64)
        _lib.check(lib.b200_tp_exchange_alloc(nbytes, ctypes.byref(mine), handle), "b200_tp_exchange_alloc")
        handles = [None] * self.world
        dist.all_gather_object(handles, handle.raw, group=self.group)
        peers = []
        for r, hb in enumerate(handles):
            if r == self.rank:
                peers.append(mine.value)
                continue
            q = ctypes.c_void_p()
            _lib.check(lib.b200_tp_exchange_open(hb, ctypes.byref(q)), "b200_tp_exchange_open")
            peers.append(q.value)
        dist.barrier(group=self.group)
        self.peers = peers
        self.nbytes = nbytes
        self.peer_array = (ctypes.c_void_p * 8)(*peers)

    def check_error(self):
        """Raise if an argmax combine gave up waiting for a peer (synchronises)."""
        if self.peers is not None:
            rc = _lib.lib().b200_tp_exchange_error(ctypes.c_void_p(self.peers[self.rank]))
            if rc != 0:
                raise _lib.B200Error(f"tensor-parallel exchange: a bounded wait for a peer gave up ({rc})")

    def reset_exchange(self):
        """After a pass that reported a timeout: zero every GPU's exchange buffer (collective; the caller also
        clears the models' error words, ``Model.check_fused_error`` does that when it raises)."""
        if self.peers is None:
            return
        import torch.distributed as dist
        torch.cuda.synchronize()
        dist.barrier(group=self.group)
        lib = _lib.lib()
        _lib.check(lib.b200_tp_exchange_reset(ctypes.c_void_p(self.peers[self.rank]), self.nbytes), "b200_tp_exchange_reset")
        dist.barrier(group=self.group)

    def close_exchange(self):
        """Unmap the peers' buffers and free this GPU's (collective: no rank may still be inside a pass)."""
        if self.peers is None:
            return
        import torch.distributed as dist
        torch.cuda.synchronize()
        dist.barrier(group=self.group)
        lib = _lib.lib()
        for r, q in enumerate(self.peers):
            if r != self.rank:
                lib.b200_tp_exchange_close(ctypes.c_void_p(q))
        dist.barrier(group=self.group)
        lib.b200_tp_exchange_free(ctypes.c_void_p(self.peers[self.rank]))
        self.peers = self.peer_array = None


def _rows(lin: "QLinear", r0: int, r1: int) -> "QLinear":
    """Output rows [r0, r1) of a linear layer (column-parallel shard)."""
    return QLinear(lin.weight[r0:r1].contiguous(), lin.scales[r0:r1].contiguous(), lin.biases[r0:r1].contiguous(),
                   None if lin.bias is None else lin.bias[r0:r1].contiguous())


def _cols(lin: "QLinear", k0: int, k1: int) -> "QLinear":
    """Input features [k0, k1) of a linear layer (row-parallel shard; k0, k1 multiples of 128)."""
    return QLinear(lin.weight[:, k0 // 8:k1 // 8].contiguous(), lin.scales[:, k0 // 64:k1 // 64].contiguous(),
                   lin.biases[:, k0 // 64:k1 // 64].contiguous(), None)


class QLinear:
    """A 4-bit quantised linear layer: packed weights, fp16 scales / biases, optional fp16 bias."""

    def __init__(self, wq, scales, biases, bias=None):
        self.weight, self.scales, self.biases, self.bias = wq, scales, biases, bias
        self.out_features = wq.shape[0]
        self.in_features = wq.shape[1] * 8
        self.group_size, self.bits = 64, 4
        self.tiled = None
        self._fast_of = None

    def relayout(self, keep_rowmajor: bool = False):
        """Build the streaming layout of this layer's weights; drop the row-major tensors unless asked.

        Passes trust what is found here about the scales for as long as ``tiled`` is the same tensor and torch has counted no change
        of it.  A write that torch does not count (through ``.data``, a view of another type made in inference mode, DLPack,
        ``__cuda_array_interface__`` or a kernel of the caller's) needs ``weights_changed()`` before the next pass: scales outside 2^-14 .. 2^-4 would be expanded wrongly."""
        self._nbytes = self.nbytes()
        self.tiled = qk.relayout(self.weight, self.scales, self.biases)
        self._look_at(self.scales)
        if not keep_rowmajor:
            self.weight = self.scales = self.biases = None

    def weights_changed(self):
        """Look at the scales of the re-laid-out weights again (waits for the device).  For a layer of a ``Model``:
        ``Model.weights_changed``, which also lets go of what was made for the old ones."""
        self._look_at(qk.tiled_scales(self.tiled, self.out_features, self.in_features))

    def _look_at(self, scales):
        # a pass's kernels expand nibbles with a shorter, bit-identical sequence when every scale's fp16
        # exponent field is in 1..10 (2^-14 <= |s| < 2^-4)
        e = (scales.view(torch.int16).to(torch.int32) >> 10) & 31
        ok = not self.tiled.is_inference() and bool(((e >= 1) & (e <= 10)).all())      # (a caller's inference tensor does not count its changes)
        self._fast_of = (self.tiled, self.tiled._version) if ok else None

    @property
    def scales_fast(self) -> bool:
        """Every scale is known to allow the short expansion: of the tensor that ``relayout`` made, neither replaced nor written since."""
        return self._fast_of is not None and self._fast_of[0] is self.tiled and self._fast_of[1] == self.tiled._version

    def nbytes(self) -> int:
        if self.weight is None:
            return self._nbytes
        n = self.weight.numel() * 4 + self.scales.numel() * 2 + self.biases.numel() * 2
        return n + (self.bias.numel() * 2 if self.bias is not None else 0)

    def __call__(self, x):
        """Stand-alone use, like ``NewQuantizedLinear.__call__`` (``mlx_model_fwd_bench.py:65-73``)."""
        return qk.matmul(x, self.weight, self.scales, self.biases, self.group_size, bias=self.bias)[0]


class FwdInputs:
    """Device-resident inputs of one forward pass (what the tree kernels write)."""

    def __init__(self, device):
        self.tokens = torch.zeros(MAX_ROWS, dtype=torch.int32, device=device)
        self.pos = torch.zeros(MAX_ROWS, dtype=torch.int32, device=device)
        self.mask = torch.zeros(MAX_ROWS, dtype=torch.int64, device=device)   # uint64 bit masks
        self.prefix = torch.zeros(MAX_REQUESTS, dtype=torch.int32, device=device)   # committed length per request
        self.last = torch.zeros(1, dtype=torch.int32, device=device)                # index of the pass's last token


class KVCache:
    """K/V of every layer in one allocation ``[layers][2][Hkv][rows][hd]`` plus the committed length.

    ``offset`` has the meaning of ``mlx_lm``'s ``KVCache.offset`` (rows in use); the reference
    rewinds it directly (``mlx_eagle.py:376,405-406,593-594``), and so may callers here.
    """

    def __init__(self, args: ModelArgs, rows: int, device, data: Optional[torch.Tensor] = None):
        self.rows = int(rows)
        self.data = data if data is not None else torch.zeros(
            args.num_hidden_layers, 2, args.num_key_value_heads, self.rows, args.head_dim,
            dtype=torch.float16, device=device)
        self.offset = 0

    def layer(self, i):
        return self.data[i, 0], self.data[i, 1]

    @property
    def state(self):
        return self.data[:, 0, :, : self.offset], self.data[:, 1, :, : self.offset]


class BatchKVCache:
    """The caches of several requests that share forward passes, in one allocation
    ``[requests][layers][2][Hkv][rows][hd]`` (the layout ``b200_forward`` takes with ``requests > 1``).
    ``slabs[r]`` is request r's cache as an ordinary :class:`KVCache` view (prompt ingestion, compaction)."""

    def __init__(self, args: ModelArgs, rows: int, device, requests: int):
        self.rows, self.requests = int(rows), int(requests)
        self.data = torch.zeros(self.requests, args.num_hidden_layers, 2, args.num_key_value_heads, self.rows,
                                args.head_dim, dtype=torch.float16, device=device)
        self.slabs = [KVCache(args, rows, device, data=self.data[r]) for r in range(self.requests)]


class _Graphs:
    """Graphs of the descriptors a model's passes repeat: at most ``KEEP``, the least recently used go first.  A descriptor holds
    every address and size of its pass, so an equal one is the same pass; making its graph takes about as long as a pass of the
    large models, so only one that has come up ``AFTER`` times while among the last ``KEEP`` gets one."""
    KEEP, AFTER = 16, 4

    def __init__(self):
        self._seen = collections.OrderedDict()           # descriptor -> [times, graph]
        self._settings = 0                               # the process's, when they were made

    def clear(self):
        while self._seen:
            _lib.lib().b200_graph_destroy(self._seen.popitem()[1][1])

    def get(self, desc, device):
        settings = _lib.lib().b200_launch_settings()
        if settings != self._settings:                   # (a graph keeps the poll limit, the plan and the launch attributes it was made with)
            self.clear()
            self._settings = settings
        key = bytes(desc)
        entry = self._seen.get(key)
        if entry is None:
            if len(self._seen) >= self.KEEP:
                _lib.lib().b200_graph_destroy(self._seen.popitem(last=False)[1][1])
            self._seen[key] = [1, None]
            return None
        self._seen.move_to_end(key)
        entry[0] += 1
        if entry[1] is None and entry[0] > self.AFTER:
            exec_ = ctypes.c_void_p()
            with torch.cuda.device(device):
                _lib.check(_lib.lib().b200_forward_graph(ctypes.byref(desc), ctypes.byref(exec_)), "b200_forward_graph")
            entry[1] = exec_.value
        return entry[1]

    def __del__(self):
        try:
            self.clear()
        except Exception:                                # (interpreter shutdown)
            pass


class Model:
    def __init__(self, args: ModelArgs, layers: List[dict], embed: QLinear, norm: torch.Tensor,
                 lm_head: Optional[QLinear], device):
        self.args = args
        self.model_type = args.model_type
        self.device = torch.device(device)
        self.layers = layers
        self.embed = embed
        self.norm = norm
        self.lm_head = lm_head if lm_head is not None else embed      # tied: as_linear (mlx_llama.py:309-310)
        inv, scaling = rope_inv_freqs(args)
        self.inv_freqs = inv.to(self.device)
        self.rope_scaling_factor = float(scaling)
        self.scale = args.head_dim ** -0.5
        H, hd = args.hidden_size, args.head_dim
        self.nq, self.nkv = args.num_attention_heads * hd, args.num_key_value_heads * hd
        f16 = dict(dtype=torch.float16, device=self.device)
        self.h = torch.zeros(MAX_ROWS, H, **f16)
        self.xn = torch.zeros(MAX_ROWS, H, **f16)
        self.qkv = torch.zeros(MAX_ROWS, self.nq + 2 * self.nkv, **f16)
        self.attn = torch.zeros(MAX_ROWS, self.nq, **f16)
        self.act = torch.zeros(MAX_ROWS, args.intermediate_size, **f16)
        self.logits = torch.zeros(MAX_ROWS, args.vocab_size, **f16)
        self._attn_ws = None
        self._attn_ws_rows = 0
        # matmul inputs of the fused forward, in a layout of its kernels: h * norm weight, attention output, MLP activations
        self.hw = torch.zeros(H // 128 * MAX_ROWS * 128 if H % 128 == 0 else 0, **f16)      # h * norm weight
        self.xt_attn = torch.zeros(self.nq // 128 * MAX_ROWS * 128 if self.nq % 128 == 0 else 0, **f16)
        self.xt_act = torch.zeros(args.intermediate_size // 128 * MAX_ROWS * 128
                                  if args.intermediate_size % 128 == 0 else 0, **f16)
        self.fused = True                                # b200_forward when possible
        self._fwd_ws = None
        self._fwd_ws_key = None
        # device pointers of the layers, and whether all allow the short expansion: kept up to date by _gather_layers()
        self._layers_host = self._layer_table = self._layers_fast = None
        self.tp: Optional[TensorParallel] = None         # set by shard(): this model is one shard of a tensor-parallel model
        self.vocab_offset = 0
        self.part32 = None
        self.timeline = None
        self.attn_split_blocks = 0                       # 0 = library default; n: split the keys from n blocks on; < 0 = always
        self.phase_mask = 0                              # profiling: run only some phase kinds (0 = all)
        self.grid_ctas = 0                               # CTAs of a shard's persistent kernel (0 = one per SM)
        self.fast_dequant = True                         # allow the short nibble expansion when every scale permits it
        self.tp_two_shot = 0                             # tensor-parallel exchange: 0 library's choice (push), 1 two-step, 2 pull behind a hierarchical barrier, 3 push, 4 pull
        self.prefill_large_m = True                      # prompts beyond 32 tokens through b200_prefill
        self._pf_buf, self._pf_fits = None, False        # buffers of that path, made on first use
        self._scales_fast, self._fuse_fits = None, False
        self._graphs = _Graphs()
        self.fwd = FwdInputs(self.device)

    # ------------------------------------------------------------------ construction
    @staticmethod
    def random_init(args: ModelArgs, seed: int, device, gen_device=None, head_rows: Optional[int] = None) -> "Model":
        """Seeded N(0, 0.02) weights quantised to 4 bit / group 64 (stands in for a checkpoint).

        ``gen_device`` is where the random numbers are drawn ("cpu" gives the same weights on any
        machine, which the parity tests use; the default draws on ``device``, which is what a
        multi-GB model needs to be built in seconds)."""
        device = torch.device(device)
        gdev = torch.device(gen_device) if gen_device is not None else device
        gen = torch.Generator(device=gdev).manual_seed(seed)
        H, I, hd = args.hidden_size, args.intermediate_size, args.head_dim
        nq, nkv = args.num_attention_heads * hd, args.num_key_value_heads * hd

        def qlin(n, k, bias=False):
            w = torch.randn(n, k, generator=gen, device=gdev) * 0.02
            wq, s, b = (t.to(device) for t in quantize(w))
            bv = (torch.randn(n, generator=gen, device=gdev) * 0.02).half().to(device) if bias else None
            return QLinear(wq, s, b, bv)

        def norm_w():
            return (1.0 + 0.1 * torch.randn(H, generator=gen, device=gdev)).half().to(device)

        layers = []
        for _ in range(args.num_hidden_layers):
            layers.append(dict(
                qkv=qlin(nq + 2 * nkv, H, bias=args.attention_bias), o=qlin(H, nq), gate=qlin(I, H), up=qlin(I, H),
                down=qlin(H, I), input_norm=norm_w(), post_norm=norm_w()))
        embed = qlin(args.vocab_size, H)
        if head_rows is not None:                       # a vocabulary shard of the head (see random_init_shard)
            lm_head = _rows(embed, 0, head_rows) if args.tie_word_embeddings else qlin(head_rows, H)
        else:
            lm_head = None if args.tie_word_embeddings else qlin(args.vocab_size, H)
        return Model(args, layers, embed, norm_w(), lm_head, device)

    @staticmethod
    def random_init_shard(args: ModelArgs, seed: int, device, rank: int, world: int, group=None,
                          shard_head: bool = True) -> "Model":
        """A tensor-parallel shard drawn directly at shard shapes, for models too large to build whole on one
        GPU.  Every rank must pass the same seed: embeddings and norms then agree across ranks (which the
        replicated hidden state needs); the shards' own weights are the same random numbers on every rank,
        which changes nothing about the work done.  Not a shard of ``random_init(args, seed)``.
        ``shard_head=False`` keeps the whole vocabulary projection on every GPU (a tensor-parallel DRAFT: its logits
        feed the tree kernels, which want every vocabulary row; only the layers are cut)."""
        import dataclasses
        a = args
        hd = a.head_dim
        if any(v % world for v in (a.num_attention_heads, a.num_key_value_heads, a.vocab_size)) or \
                (a.intermediate_size // world) % 128 or (a.num_attention_heads * hd // world) % 128 or \
                (a.vocab_size // world) % 8:
            raise _lib.B200Error("heads, kv heads, MLP width (in multiples of 128) and vocabulary must divide by the TP degree")
        largs = dataclasses.replace(a, num_attention_heads=a.num_attention_heads // world,
                                    num_key_value_heads=a.num_key_value_heads // world,
                                    intermediate_size=a.intermediate_size // world)
        m = Model.random_init(largs, seed, device, head_rows=a.vocab_size // world if shard_head else None)
        m.tp = TensorParallel(rank, world, group)
        m.vocab_offset = rank * (a.vocab_size // world) if shard_head else 0
        m.part32 = torch.zeros(MAX_ROWS, a.hidden_size, dtype=torch.float32, device=m.device)
        return m

    def shard(self, rank: int, world: int, group=None, shard_head: bool = True) -> "Model":
        """This model's shard ``rank`` of ``world`` for tensor-parallel execution (call before ``relayout``).
        Heads, kv heads, MLP rows and vocabulary rows are cut evenly; embeddings and norms are replicated.
        ``shard_head=False`` leaves the vocabulary projection whole on every GPU (for a tensor-parallel draft)."""
        a = self.args
        if any(v % world for v in (a.num_attention_heads, a.num_key_value_heads, a.vocab_size)) or \
                (a.intermediate_size // world) % 128 or (self.nq // world) % 128 or (a.vocab_size // world) % 8:
            raise _lib.B200Error("heads, kv heads, MLP width (in multiples of 128) and vocabulary must divide by the TP degree")
        nq, nkv, I, V = self.nq // world, self.nkv // world, a.intermediate_size // world, a.vocab_size // world
        layers = []
        for lw in self.layers:
            q = lw["qkv"]
            if q.weight is None:
                raise _lib.B200Error("shard() needs the row-major weights: call it before relayout()")
            parts = [_rows(q, rank * nq, (rank + 1) * nq),
                     _rows(q, self.nq + rank * nkv, self.nq + (rank + 1) * nkv),
                     _rows(q, self.nq + self.nkv + rank * nkv, self.nq + self.nkv + (rank + 1) * nkv)]
            qkv = QLinear(torch.cat([p_.weight for p_ in parts]), torch.cat([p_.scales for p_ in parts]),
                          torch.cat([p_.biases for p_ in parts]),
                          None if q.bias is None else torch.cat([p_.bias for p_ in parts]))
            layers.append(dict(qkv=qkv, o=_cols(lw["o"], rank * nq, (rank + 1) * nq),
                               gate=_rows(lw["gate"], rank * I, (rank + 1) * I), up=_rows(lw["up"], rank * I, (rank + 1) * I),
                               down=_cols(lw["down"], rank * I, (rank + 1) * I),
                               input_norm=lw["input_norm"], post_norm=lw["post_norm"]))
        import dataclasses
        largs = dataclasses.replace(a, num_attention_heads=a.num_attention_heads // world,
                                    num_key_value_heads=a.num_key_value_heads // world, intermediate_size=I)
        head = _rows(self.lm_head, rank * V, (rank + 1) * V) if shard_head else (None if self.lm_head is self.embed else self.lm_head)
        m = Model(largs, layers, self.embed, self.norm, head, self.device)
        m.tp = TensorParallel(rank, world, group)
        m.vocab_offset = rank * V if shard_head else 0
        m.part32 = torch.zeros(MAX_ROWS, a.hidden_size, dtype=torch.float32, device=self.device)
        return m

    def greedy_token(self, logits_row: torch.Tensor) -> int:
        """Argmax of one row of logits over the whole vocabulary (ties to the lower id); under tensor
        parallelism every GPU holds a slice and the slices' (max, argmax) pairs are gathered."""
        v, i = torch.max(logits_row.float(), dim=-1)
        if self.tp is None:
            return int(i)
        import torch.distributed as dist
        mine = torch.stack([v.double(), (i + self.vocab_offset).double()])
        allv = [torch.zeros_like(mine) for _ in range(self.tp.world)]
        dist.all_gather(allv, mine, group=self.tp.group)
        best = max(allv, key=lambda t: (float(t[0]), -float(t[1])))
        return int(best[1])

    @property
    def vocab_local(self) -> int:
        """Vocabulary rows this model's head produces (all of them unless it is a tensor-parallel shard)."""
        return self.lm_head.out_features

    def state_numpy(self) -> dict:
        """All weights as numpy arrays (packed weights as uint32), for a CPU checker."""
        import numpy as np

        def lin(q: QLinear):
            d = dict(weight=q.weight.cpu().numpy().view(np.uint32), scales=q.scales.cpu().numpy(),
                     biases=q.biases.cpu().numpy())
            d["bias"] = q.bias.cpu().numpy() if q.bias is not None else None
            return d

        layers = []
        for L in self.layers:
            layers.append({k: (lin(v) if isinstance(v, QLinear) else v.cpu().numpy()) for k, v in L.items()})
        return dict(layers=layers, embed=lin(self.embed), norm=self.norm.cpu().numpy(),
                    lm_head=None if self.lm_head is self.embed else lin(self.lm_head),
                    inv_freqs=self.inv_freqs.cpu().numpy(), rope_scaling_factor=self.rope_scaling_factor)

    def linear_weight_bytes(self) -> int:
        """Bytes of quantised weights one forward pass streams (all layers + lm_head)."""
        n = 0
        for L in self.layers:
            n += sum(L[k].nbytes() for k in ("qkv", "o", "gate", "up", "down"))
        return n + self.lm_head.nbytes()

    def make_cache(self, rows: int) -> KVCache:
        return KVCache(self.args, rows, self.device)

    def make_batch_cache(self, rows: int, requests: int) -> BatchKVCache:
        return BatchKVCache(self.args, rows, self.device, requests)

    def relayout(self):
        """Re-lay-out every linear layer for the streaming kernel (one-off, at load time).  The
        embedding keeps its row-major form, which the token gather needs."""
        for lw in self.layers:
            for k in ("qkv", "o", "gate", "up", "down"):
                lw[k].relayout()
        self.lm_head.relayout(keep_rowmajor=self.lm_head is self.embed)
        return self

    def _linear(self, x, lin: QLinear, y, M, epilogue, lin2: Optional[QLinear] = None, extra=None):
        L, p = _lib.lib(), _lib.ptr
        ws = qk.workspace(self.device)
        st = _lib.stream_ptr(self.device)
        if lin.tiled is not None:
            rc = L.b200_qmm_tiled(p(x), p(lin.tiled), p(lin2.tiled) if lin2 is not None else None, p(lin.bias),
                                  p(extra), p(y), M, lin.out_features, lin.in_features, epilogue, p(ws), ws.numel(), st)
            _lib.check(rc, "b200_qmm_tiled")
        else:
            l2 = lin2
            rc = L.b200_qmm_fused(p(x), p(lin.weight), p(lin.scales), p(lin.biases),
                                  p(l2.weight) if l2 else None, p(l2.scales) if l2 else None,
                                  p(l2.biases) if l2 else None, p(lin.bias), p(extra), p(y), M, lin.out_features,
                                  lin.in_features, 64, 0, epilogue, p(ws), ws.numel(), st)
            _lib.check(rc, "b200_qmm_fused")

    @property
    def launches_per_forward(self) -> int:
        """Launches of one pass from Python: 1 (``b200_forward``) or 9 per layer + embedding, final norm, head."""
        return 1 if self.can_fuse() else 9 * self.args.num_hidden_layers + 3

    @property
    def kernels_per_forward(self) -> int:
        """Kernels of one pass: the five per layer of the chain, embedding and head (one more where the last row tiles of a wide
        layer run as a launch of their own, not counted), the persistent kernel of a shard, or the per-op launches."""
        return 5 * self.args.num_hidden_layers + 2 if self.can_fuse() and self.tp is None else self.launches_per_forward

    # ------------------------------------------------------------------ fused forward (one native call)
    def can_fuse(self) -> bool:
        """True when the pass can run as one call of ``b200_forward``: every linear
        layer in the streaming layout, the embedding still row-major, sizes in multiples of 128."""
        if not self.fused or os.environ.get("B200_FUSED_FORWARD", "1") == "0":
            return False
        if self.tp is not None and (self.tp.peers is None or self.tp.world > 8):
            return False                         # a shard fuses once open_exchange() has mapped the peers' buffers
        if not self._fuse_fits:
            a = self.args
            if any(lw[k].tiled is None for lw in self.layers for k in ("qkv", "o", "gate", "up", "down")):
                return False
            self._fuse_fits = (a.hidden_size % 128 == 0 and a.hidden_size <= 8192 and a.intermediate_size % 128 == 0
                               and self.nq % 128 == 0 and a.head_dim in (64, 128) and a.vocab_size % 8 == 0
                               and self.vocab_local % 8 == 0)
        return self._fuse_fits and self.lm_head.tiled is not None and self.embed.weight is not None and self._gather_layers()

    def _gather_layers(self) -> bool:
        """The layers' device pointers as they are now (ahead of every pass: any tensor may have been replaced since the last).
        False if a layer has no re-laid-out weights."""
        n = self.args.num_hidden_layers
        if self._layers_host is None:
            self._layers_host, self._layers_fast = (ctypes.c_void_p * (8 * n))(), ctypes.c_uint32()
        state = _lib.ops().layer_pointers(self.layers, ctypes.addressof(self._layers_host),
                                          ctypes.addressof(self._layers_fast)) if len(self.layers) == n else -1
        if state == 0 and self._layer_table is not None:
            return True
        self._graphs.clear()                             # (a graph has the layers' pointers in it)
        self._layer_table = None
        if state < 0:
            self._fuse_fits = self._pf_fits = False
            return False
        self._layer_table = torch.tensor([p or 0 for p in self._layers_host], dtype=torch.int64).to(self.device)
        return True

    def weights_changed(self):
        """To be called between passes once re-laid-out weights have been written in a way that torch does not count (``.data``, DLPack,
        ``__cuda_array_interface__``, a kernel of the caller's).  Their scales are looked at again, which waits for the device;
        decoders capture their step anew with the next request if the outcome is another one."""
        for q in [lw[k] for lw in self.layers for k in ("qkv", "o", "gate", "up", "down")] + [self.lm_head]:
            if q.tiled is not None:
                q.weights_changed()

    def weight_addresses(self) -> bytes:
        """Where this model's weights are now, and whether they allow the short expansion, for whoever keeps graphs of its passes."""
        linears, others = [self.embed, self.lm_head], [self.norm, self.inv_freqs]
        layers = b""
        if self.can_fuse():
            layers = bytes(self._layers_host) + bytes([bool(self._layers_fast.value and self.lm_head.scales_fast and self.fast_dequant)])
        else:
            linears += [lw[k] for lw in self.layers for k in ("qkv", "o", "gate", "up", "down")]
            others += [lw[k] for lw in self.layers for k in ("input_norm", "post_norm")]
        others += [t for q in linears for t in (q.weight, q.scales, q.biases, q.bias, q.tiled)]
        return layers + repr([None if t is None else t.data_ptr() for t in others]).encode()

    def _fused_desc(self, M, cache, write_off, tail, fwd, rows, row_index, requests=1, logits=None):
        """The descriptor of ``b200_forward`` (after ``can_fuse()``, which brings the layers' pointers up to date)."""
        p = lambda t: None if t is None else t.data_ptr()
        a, d = self.args, _lib.ForwardDesc()
        d.M, d.rows_out, d.hidden, d.intermediate, d.n_heads, d.n_kv_heads = M, rows, a.hidden_size, a.intermediate_size, \
            a.num_attention_heads, a.num_key_value_heads
        d.head_dim, d.vocab, d.n_layers = a.head_dim, a.vocab_size, a.num_hidden_layers
        d.cache_rows, d.write_off, d.tail, d.requests = cache.rows, write_off, tail, requests
        d.rms_eps, d.rope_scaling, d.attn_scale = float(a.rms_norm_eps), self.rope_scaling_factor, self.scale
        d.tokens, d.pos, d.mask, d.prefix = p(fwd.tokens), p(fwd.pos), p(fwd.mask), p(fwd.prefix)
        d.row_index, d.logits, d.kv_cache = p(row_index), p(self.logits if logits is None else logits), p(cache.data)
        d.inv_freq = p(self.inv_freqs)
        d.embed_wq, d.embed_scales, d.embed_biases = p(self.embed.weight), p(self.embed.scales), p(self.embed.biases)
        d.final_norm, d.lm_head_tiled, d.layer_table = p(self.norm), p(self.lm_head.tiled), p(self._layer_table)
        d.h, d.hw, d.qkv, d.attn, d.act = p(self.h), p(self.hw), p(self.qkv), p(self.xt_attn), p(self.xt_act)
        d.grid_ctas, d.phase_mask, d.attn_split_blocks = self.grid_ctas, self.phase_mask, self.attn_split_blocks
        self._scales_fast = bool(self._layers_fast.value and self.lm_head.scales_fast)
        d.scales_in_fast_range = 1 if (self._scales_fast and self.fast_dequant) else 0
        if self.tp is not None:
            d.tp_world, d.tp_rank, d.head_rows = self.tp.world, self.tp.rank, self.vocab_local
            d.tp_two_shot = self.tp_two_shot
            for r, q in enumerate(self.tp.peers):
                d.tp_peers[r] = q
        key = (cache.rows, self.grid_ctas) if self.tp is not None else 0      # (only a shard's scratch depends on them)
        if self._fwd_ws is None or self._fwd_ws_key != key:
            d32 = _lib.ForwardDesc.from_buffer_copy(d)
            d32.M, d32.rows_out, d32.write_off, d32.tail, d32.requests = MAX_ROWS, MAX_ROWS, 0, MAX_TAIL, 1
            nbytes = _lib.lib().b200_forward_workspace_bytes(ctypes.byref(d32))
            if nbytes == 0:
                raise _lib.B200Error("b200_forward_workspace_bytes rejected the model shape")
            self._fwd_ws = torch.zeros(nbytes, dtype=torch.uint8, device=self.device)
            self._fwd_ws_key = key
        d.workspace, d.workspace_bytes = p(self._fwd_ws), self._fwd_ws.numel()
        if self.tp is None:
            d.timeline, d.timeline_pitch = ctypes.addressof(self._layers_host), _lib.LAYERS_ON_HOST
        elif self.timeline is not None:
            d.timeline, d.timeline_pitch = p(self.timeline), self.timeline.shape[1]
        return d

    def enable_timeline(self, on: bool = True):
        """Profiling hook of a shard's persistent kernel: per SM, the device timer (ns) at arrival at and
        departure from every device-wide barrier of the next pass, plus six stamps inside the matmul phase
        that ends at the barrier: entry, rstd done, first stage landed, stages done, K-parts reduced, end
        (``self.timeline`` int64 ``[SMs, barriers + 1, 8]``; the last entry holds the end of the kernel)."""
        if on:
            if self.tp is None:
                raise _lib.B200Error("the timeline is of a shard's persistent kernel: without tensor parallelism a pass is a "
                                     "chain of kernels (time them with a profiler or CUDA events)")
            sms = torch.cuda.get_device_properties(self.device).multi_processor_count
            self.timeline = torch.zeros(sms, 10 * self.args.num_hidden_layers + 2, 8, dtype=torch.int64, device=self.device)
        else:
            self.timeline = None

    def check_fused_error(self):
        """Raise if a bounded wait inside ``b200_forward``, ``b200_prefill`` or a matmul of the per-op path ever ran out
        (synchronises)."""
        if self._fwd_ws is not None:
            code = int(self._fwd_ws[:16].view(torch.int32)[2])
            if code != 0:
                self._fwd_ws[:4352].zero_()
                raise _lib.B200Error(f"b200_forward: a bounded wait gave up inside the kernel (code {code})")
        if self._pf_buf is not None:
            word = self._pf_buf["ws"][4092:4096].view(torch.int32)
            code = int(word)
            if code != 0:
                word.zero_()
                raise _lib.B200Error(f"b200_prefill: a bounded wait ran out inside a kernel of the pass (code {code})")
        if not self.can_fuse():
            code = qk.stream_error(self.device)
            if code != 0:
                qk.workspace(self.device)[4092:4096].zero_()
                raise _lib.B200Error(f"a bounded wait ran out inside a matmul (code {code})")
        if self.tp is not None:
            self.tp.check_error()

    def _row_parallel(self, x, lin: QLinear, M: int):
        """h += x . W^T for o_proj / down_proj.  Under tensor parallelism W holds this GPU's K shard: the fp32
        partial product is all-reduced (NCCL over NVLink), then added to the residual with the rounding points
        of the unsharded epilogue."""
        if self.tp is None:
            self._linear(x, lin, self.h, M, qk.EPI_RESIDUAL, extra=self.h)
            return
        if lin.tiled is None:
            raise _lib.B200Error("tensor-parallel layers need the streaming layout: call relayout() after shard()")
        self._linear(x, lin, self.part32, M, qk.EPI_F32)
        part = self.part32[:M]
        self.tp.all_reduce_sum(part)
        _lib.check(_lib.lib().b200_residual_add_f32(_lib.ptr(self.h), _lib.ptr(part), M, self.args.hidden_size,
                                                    _lib.stream_ptr(self.device)), "b200_residual_add_f32")

    # ------------------------------------------------------------------ device-side forward
    def _attention_workspace(self, cache: KVCache):
        if self._attn_ws is None or self._attn_ws_rows < cache.rows:
            a = self.args
            nbytes = _lib.lib().b200_tree_attention_workspace_bytes(
                MAX_ROWS, a.num_attention_heads, a.num_key_value_heads, a.head_dim, cache.rows)
            self._attn_ws = torch.zeros(nbytes, dtype=torch.uint8, device=self.device)
            self._attn_ws_rows = cache.rows
        return self._attn_ws

    def _run_fused(self, desc):
        """``b200_forward``, or the graph of a descriptor that has come up ``_Graphs.AFTER`` times: a decode loop repeats one or two
        (the result's address alternates), and a launch of the graph is 120 launches less."""
        lib, stream = _lib.lib(), _lib.stream_ptr(self.device)
        if self.tp is None and not torch.cuda.is_current_stream_capturing():
            exec_ = self._graphs.get(desc, self.device)
            if exec_ is not None:
                _lib.check(lib.b200_graph_launch(exec_, stream), "b200_graph_launch")
                return
        _lib.check(lib.b200_forward(ctypes.byref(desc), stream), "b200_forward")

    def forward_device(self, M: int, cache: KVCache, write_off: int, tail: int, fwd: Optional[FwdInputs] = None,
                       logits_rows: Optional[int] = None, row_index: Optional[torch.Tensor] = None, requests: int = 1):
        """One forward pass of ``M`` tokens whose ids / positions / masks / committed length sit in
        ``fwd`` (device memory).  New K/V rows go to cache row ``prefix + write_off + m``; query m sees
        rows ``< prefix`` and tail row j iff bit j of ``fwd.mask[m]``.  Returns fp16 logits
        ``(logits_rows or M, V)`` (a view of an internal buffer); with ``row_index`` (device int) only
        rows ``row_index .. row_index+logits_rows-1`` of the hidden state reach the head."""
        return self._forward(M, cache, write_off, tail, fwd, logits_rows, row_index, requests)

    def _forward(self, M, cache, write_off, tail, fwd=None, logits_rows=None, row_index=None, requests=1, out=None):
        """``forward_device`` into ``out`` (contiguous fp16, its rows of this model's share of the vocabulary), or into the
        model's own buffer."""
        if not (1 <= M <= MAX_ROWS and 1 <= tail <= MAX_TAIL and write_off + M // requests <= tail):
            raise _lib.B200Error("forward_device: need 1 <= M <= 32, tail <= 64, write_off + M <= tail")
        fwd = fwd or self.fwd
        if requests > 1:
            # several requests share the pass (and every weight read): M = requests x rows of each; ``cache`` is a
            # BatchKVCache, fwd.prefix / row_index hold one entry per request, logits come back as
            # [requests * logits_rows][V]
            if not (self.can_fuse() and isinstance(cache, BatchKVCache) and cache.requests == requests
                    and M % requests == 0 and self.tp is None):
                raise _lib.B200Error("forward_device: several requests need relayouted weights and a BatchKVCache")
            rows = M // requests if logits_rows is None else logits_rows
            desc = self._fused_desc(M, cache, write_off, tail, fwd, rows, row_index, requests, out)
            _lib.check(_lib.lib().b200_forward(ctypes.byref(desc), _lib.stream_ptr(self.device)), "b200_forward")
            return self.logits[: requests * rows] if out is None else out
        if self.can_fuse():
            rows = M if logits_rows is None else logits_rows
            self._run_fused(self._fused_desc(M, cache, write_off, tail, fwd, rows, row_index, logits=out))
            if out is not None:
                return out
            vl = self.vocab_local
            return self.logits[:rows] if vl == self.args.vocab_size else self.logits.view(-1)[: rows * vl].view(rows, vl)
        a, L, lib = self.args, _lib.lib(), _lib.lib()
        st, p = _lib.stream_ptr(self.device), _lib.ptr
        ws = qk.workspace(self.device)
        aws = self._attention_workspace(cache)
        H, I, hd = a.hidden_size, a.intermediate_size, a.head_dim
        Hq, Hkv = a.num_attention_heads, a.num_key_value_heads
        nqkv = self.nq + 2 * self.nkv
        eps = float(a.rms_norm_eps)
        ck = _lib.check
        ck(L.b200_embed_gather(p(fwd.tokens), p(self.embed.weight), p(self.embed.scales), p(self.embed.biases),
                               p(self.h), M, H, a.vocab_size, st), "b200_embed_gather")
        for li, lw in enumerate(self.layers):
            kc, vc = cache.layer(li)
            ck(L.b200_rms_norm(p(self.h), p(lw["input_norm"]), p(self.xn), None, M, H, eps, st), "b200_rms_norm")
            self._linear(self.xn, lw["qkv"], self.qkv, M, qk.EPI_NONE)
            ck(L.b200_rope_kv_append(p(self.qkv), p(fwd.pos), p(self.inv_freqs), self.rope_scaling_factor, p(kc),
                                     p(vc), p(fwd.prefix), write_off, M, Hq, Hkv, hd, cache.rows, st), "rope")
            ck(L.b200_tree_attention(p(self.qkv), nqkv, p(kc), p(vc), p(fwd.mask), p(fwd.prefix), tail,
                                     p(self.attn), M, Hq, Hkv, hd, cache.rows, cache.rows, self.scale,
                                     p(aws), aws.numel(), st), "b200_tree_attention")
            self._row_parallel(self.attn, lw["o"], M)
            ck(L.b200_rms_norm(p(self.h), p(lw["post_norm"]), p(self.xn), None, M, H, eps, st), "b200_rms_norm")
            self._linear(self.xn, lw["gate"], self.act, M, qk.EPI_SILU_MUL, lin2=lw["up"])
            self._row_parallel(self.act, lw["down"], M)
        rows = M if logits_rows is None else logits_rows
        ck(L.b200_rms_norm(p(self.h), p(self.norm), p(self.xn), p(row_index), rows, H, eps, st), "final norm")
        self._linear(self.xn, self.lm_head, self.logits if out is None else out, rows, qk.EPI_NONE)
        if out is not None:
            return out
        vl = self.vocab_local                      # a tensor-parallel shard produces its slice of the vocabulary
        return self.logits[:rows] if vl == a.vocab_size else self.logits.view(-1)[: rows * vl].view(rows, vl)

    # ------------------------------------------------------------------ prompt ingestion, one weight read per 128 rows
    def can_prefill_large_m(self) -> bool:
        """True when a causal prompt can go through ``b200_prefill``: weights in the streaming layout, sizes it takes, no
        tensor-parallel shard."""
        if not self.prefill_large_m or self.tp is not None or os.environ.get("B200_PREFILL_LARGE_M", "1") == "0":
            return False
        if not self._pf_fits:
            a = self.args
            lins = [lw[k] for lw in self.layers for k in ("qkv", "o", "gate", "up", "down")] + [self.lm_head]
            self._pf_fits = (all(q.tiled is not None for q in lins) and self.embed.weight is not None
                             and all(q.out_features % 8 == 0 and q.in_features % 128 == 0 for q in lins)
                             and a.hidden_size <= 8192 and a.head_dim in (64, 128))
        return self._pf_fits and self.lm_head.tiled is not None and self.embed.weight is not None and self._gather_layers()

    def _prefill_large_m(self, tokens: torch.Tensor, cache: KVCache, off: int, logits: Optional[torch.Tensor], rows: int):
        """One causal pass of up to ``PREFILL_ROWS`` prompt tokens (device int32) starting at cache row ``off``
        (``mlx_eagle.py:522-535`` ingests the prompt in chunks; ``mlx_llama.py:231-249`` is the layer), launched from native
        code (``b200_prefill``).  Writes the logits of all tokens (``rows`` = their count) or of the last (``rows`` = 1) to
        ``logits``; ``rows`` = 0: cache rows only."""
        p = lambda t: t.data_ptr()
        a, d, buf = self.args, _lib.PrefillDesc(), self._pf_buf
        H, I = a.hidden_size, a.intermediate_size
        if buf is None:
            R, f16 = PREFILL_ROWS, dict(dtype=torch.float16, device=self.device)
            buf = dict(h=torch.empty(R, H, **f16), xn=torch.empty(R, H, **f16),
                       qkv=torch.empty(R, self.nq + 2 * self.nkv, **f16), attn=torch.empty(R, self.nq, **f16),
                       act=torch.empty(R, I, **f16), ws=torch.zeros(4096 + (16 << 20), dtype=torch.uint8, device=self.device))
            self._pf_buf = buf
        d.hidden, d.intermediate, d.n_heads, d.n_kv_heads = H, I, a.num_attention_heads, a.num_key_value_heads
        d.head_dim, d.vocab, d.n_layers = a.head_dim, a.vocab_size, a.num_hidden_layers
        d.rms_eps, d.rope_scaling, d.attn_scale = float(a.rms_norm_eps), self.rope_scaling_factor, self.scale
        d.inv_freq, d.final_norm, d.lm_head_tiled = p(self.inv_freqs), p(self.norm), p(self.lm_head.tiled)
        d.embed_wq, d.embed_scales, d.embed_biases = p(self.embed.weight), p(self.embed.scales), p(self.embed.biases)
        d.layers = ctypes.addressof(self._layers_host)   # (brought up to date by can_prefill_large_m())
        d.h, d.xn, d.qkv, d.attn, d.act = (p(buf[k]) for k in ("h", "xn", "qkv", "attn", "act"))
        d.workspace, d.workspace_bytes = p(buf["ws"]), buf["ws"].numel()
        d.n, d.off, d.cache_rows, d.kv_cache, d.tokens = tokens.numel(), off, cache.rows, p(cache.data), p(tokens)
        d.head_out = 0 if rows == 0 else (1 if rows == d.n and rows > 1 else 2)
        d.logits = p(logits) if rows else None
        _lib.check(_lib.lib().b200_prefill(ctypes.byref(d), _lib.stream_ptr(self.device)), "b200_prefill")

    # ------------------------------------------------------------------ reference-style call
    def __call__(self, inputs: torch.Tensor, cache: Optional[KVCache] = None, mask: Optional[torch.Tensor] = None,
                 position_ids: Optional[Union[torch.Tensor, int]] = None, flat_rope: bool = False,
                 logits_last_only: bool = False) -> torch.Tensor:
        """``logits (1, L, V)``; the argument meanings follow ``mlx_llama.py:298-313`` / ``:121-196``.

        ``mask`` is the additive matrix ``(1,1,L,cache.offset+L)`` of 0 / -inf the reference passes
        (``mlx_eagle.py:177,338``); ``None`` means causal.  Calls longer than 32 tokens (prompt ingestion) are split
        into passes of 1024 (``b200_prefill``) or, where that does not apply, 32, which is only possible with the causal mask.
        ``logits_last_only`` (an addition) returns only the last token's logits ``(1, 1, V)``.
        """
        if cache is None:
            raise _lib.B200Error("a KVCache is required (the reference's cache-less branch is not on this path)")
        inputs = inputs.reshape(-1)
        Ltot = inputs.numel()
        if Ltot == 0:
            raise _lib.B200Error("no tokens")
        if Ltot > MAX_ROWS and (mask is not None or position_ids is not None):
            raise _lib.B200Error("explicit masks / positions are limited to 32 tokens per call")
        if Ltot > MAX_ROWS and self.can_prefill_large_m():
            inputs = inputs.to(self.device, torch.int32).contiguous()
            out = torch.empty(1 if logits_last_only else Ltot, self.args.vocab_size, dtype=torch.float16, device=self.device)
            for c0 in range(0, Ltot, PREFILL_ROWS):
                chunk = inputs[c0:c0 + PREFILL_ROWS]
                off, n = cache.offset, chunk.numel()
                if off + n > cache.rows:
                    raise _lib.B200Error("KV cache is full")
                if logits_last_only:
                    self._prefill_large_m(chunk, cache, off, out, 1 if c0 + n >= Ltot else 0)
                else:
                    self._prefill_large_m(chunk, cache, off, out[c0:c0 + n], n)
                cache.offset = off + n
            return out.unsqueeze(0)
        inputs = self._ids(inputs)
        out = torch.empty(1 if logits_last_only else Ltot, self.vocab_local, dtype=torch.float16, device=self.device)
        for c0 in range(0, Ltot, MAX_ROWS):
            chunk = inputs[c0:c0 + MAX_ROWS]
            L = chunk.numel()
            off = cache.offset
            if off + L > cache.rows:
                raise _lib.B200Error("KV cache is full")
            if position_ids is None:
                pos, base, step = None, off, 1
            elif isinstance(position_ids, int):
                pos, base, step = None, position_ids, 0 if flat_rope else 1
            else:
                pos, base, step = position_ids, 0, 0
            prefix, write_off, tail, vis = off, 0, L, None
            if mask is not None:
                shown = (mask.reshape(L, -1).float().cpu() == 0)
                cols = shown.shape[1]
                if cols != off + L:
                    raise _lib.B200Error("mask must have cache.offset + L columns")
                hidden = (~shown.all(dim=0)).nonzero()
                first_hidden = int(hidden[0]) if hidden.numel() else cols
                prefix = max(min(first_hidden, off), cols - MAX_TAIL)
                if not bool(shown[:, :prefix].all()):
                    raise _lib.B200Error("mask hides a column more than 64 rows before the end of the cache")
                tail, write_off = cols - prefix, off - prefix
                # bit j = tail row j (bit 63 is the sign: distinct powers of two add up without a carry)
                vis = (shown[:, prefix:].to(torch.int64) << torch.arange(tail, dtype=torch.int64)).sum(dim=1)
            self._pass(chunk, cache, prefix, write_off, tail, pos, base, step, vis, out if logits_last_only else out[c0:c0 + L])
            cache.offset = off + L
        return out.unsqueeze(0)

    def _ids(self, t: torch.Tensor) -> torch.Tensor:
        """Token ids or positions as the device takes them: int32 or int64, flat, on the model's device."""
        t = t.reshape(-1)
        return t.to(self.device, t.dtype if t.dtype in (torch.int32, torch.int64) else torch.int32).contiguous()

    def _pass(self, tokens, cache, prefix, write_off, tail, pos, pos_base, pos_step, vis, out):
        """Inputs and launch of one pass of up to 32 tokens.  ``vis``: None = causal, int64 mask words, or the visibility of
        the pass's own tokens to each other, bool or additive fp32 ``(L, L)``.  ``out``: the logits of all tokens, or of the
        last (one row)."""
        f, L = self.fwd, tokens.numel()
        pp, pos64, stride, vp, kind = None, 0, 1, None, 0
        if pos is not None:
            pos = self._ids(pos)
            if pos.numel() not in (1, L):
                raise _lib.B200Error(f"{pos.numel()} positions for {L} tokens")
            pp, pos64, stride = pos.data_ptr(), pos.dtype == torch.int64, 0 if pos.numel() == 1 else 1
        if vis is not None:
            if vis.dtype == torch.int64:
                f.mask[:L].copy_(vis)
                kind = -1
            else:
                vp, kind = vis.data_ptr(), 1 if vis.dtype == torch.bool else 2
        _lib.check(_lib.lib().b200_pass_inputs(tokens.data_ptr(), tokens.dtype == torch.int64, pp, pos64, stride, pos_base, pos_step, vp,
                                               kind, L, prefix, f.tokens.data_ptr(), f.pos.data_ptr(), f.mask.data_ptr(),
                                               f.prefix.data_ptr(), MAX_REQUESTS, f.last.data_ptr(), _lib.stream_ptr(self.device)),
                   "b200_pass_inputs")
        rows = out.shape[0]
        self._forward(L, cache, write_off, tail, f, rows, f.last if rows < L else None, out=out)

    def tree_pass(self, tokens: torch.Tensor, visible: torch.Tensor, positions: torch.Tensor, offset: int, cache: KVCache):
        """Logits ``(1, L, V)`` of a token tree behind ``cache.offset`` committed rows: token m sees those and the tokens that
        row m of ``visible`` (bool, or additive 0 / -inf) shows it, at position ``positions[m] + offset``.  Nothing is read back."""
        tokens, L = self._ids(tokens), tokens.numel()
        if cache.offset + L > cache.rows:
            raise _lib.B200Error("KV cache is full")
        visible = visible.to(self.device, torch.bool if visible.dtype == torch.bool else torch.float32).contiguous()
        out = torch.empty(L, self.vocab_local, dtype=torch.float16, device=self.device)
        self._pass(tokens, cache, cache.offset, 0, L, positions, offset, 0, visible, out)
        cache.offset += L
        return out.unsqueeze(0)


def shape_preset(name: str) -> ModelArgs:
    """Architectures named by the benchmark configurations (random-init stand-ins for checkpoints)."""
    presets = {
        "qwen2-0.5b": dict(model_type="qwen2", hidden_size=896, num_hidden_layers=24, intermediate_size=4864,
                           num_attention_heads=14, num_key_value_heads=2, head_dim=64, vocab_size=151936,
                           rms_norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=True),
        "qwen2-7b": dict(model_type="qwen2", hidden_size=3584, num_hidden_layers=28, intermediate_size=18944,
                         num_attention_heads=28, num_key_value_heads=4, head_dim=128, vocab_size=152064,
                         rms_norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=False),
        "llama3.2-1b": dict(model_type="llama", hidden_size=2048, num_hidden_layers=16, intermediate_size=8192,
                            num_attention_heads=32, num_key_value_heads=8, head_dim=64, vocab_size=128256,
                            rms_norm_eps=1e-5, rope_theta=5e5, tie_word_embeddings=True),
        "llama3-8b": dict(model_type="llama", hidden_size=4096, num_hidden_layers=32, intermediate_size=14336,
                          num_attention_heads=32, num_key_value_heads=8, head_dim=128, vocab_size=128256,
                          rms_norm_eps=1e-5, rope_theta=5e5, tie_word_embeddings=False),
        "llama3-70b": dict(model_type="llama", hidden_size=8192, num_hidden_layers=80, intermediate_size=28672,
                           num_attention_heads=64, num_key_value_heads=8, head_dim=128, vocab_size=128256,
                           rms_norm_eps=1e-5, rope_theta=5e5, tie_word_embeddings=False),
        # small shapes for tests (same structure, seconds on a CPU oracle)
        "tiny-qwen2": dict(model_type="qwen2", hidden_size=256, num_hidden_layers=2, intermediate_size=512,
                           num_attention_heads=4, num_key_value_heads=2, head_dim=64, vocab_size=1024,
                           rms_norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=True),
        "tiny-llama": dict(model_type="llama", hidden_size=512, num_hidden_layers=2, intermediate_size=1024,
                           num_attention_heads=4, num_key_value_heads=1, head_dim=128, vocab_size=2048,
                           rms_norm_eps=1e-5, rope_theta=5e5, tie_word_embeddings=False),
    }
    if name not in presets:
        raise KeyError(f"unknown shape preset {name!r}; known: {sorted(presets)}")
    return ModelArgs(**presets[name])
