"""Recurrent states of served Mamba-2 sequences and the decode step that advances them in place (``csrc/mamba_step.cu``).

A sequence's states of all layers are one block of memory, which only this module sees. Whoever looks a sequence up in
``SequenceStates`` gets the list of per-layer {"conv", "ssm"} dicts that the model's own forward takes, and the sequence leaves its
block: what was handed out is never written again, so it can be kept, shared between sequences or put back.
"""
from __future__ import annotations

import ctypes as C

import torch
import torch.nn.functional as F
from torch.nn.modules import module as torch_module

from ..models.mamba2 import Mamba2ForCausalLM, Mamba2Layer
from ..nn.modules import Embedding, Linear, RMSNorm
from ..nn.ssm import Mamba2Block
from ..ops import _lib, debug
from ..ops.gemm import gemm

MAX_ROWS = 128       # rows that the weight-streaming product takes; a larger batch goes through the model's forward


class _Block:
    """ssm [layers, H, P, N] fp32 and two buffers of convolution inputs [2, layers, taps - 1, channels]: a step reads one of them and
    writes the other."""

    __slots__ = ("ssm", "conv", "cur")

    def __init__(self, ssm, conv):
        self.ssm, self.conv, self.cur = ssm, conv, 0

    def layers(self):
        return [{"conv": self.conv[self.cur, i:i + 1], "ssm": self.ssm[i:i + 1]} for i in range(self.ssm.shape[0])]


class SequenceStates(dict):
    """States by sequence id. Reading an entry turns a block into the ordinary list; ``entry`` does not."""

    entry = dict.get

    def _open(self, sid):
        v = dict.get(self, sid)
        if isinstance(v, _Block):
            dict.__setitem__(self, sid, v.layers())

    def _open_all(self):
        for sid in list(dict.keys(self)):
            self._open(sid)
        return self

    def __getitem__(self, sid):
        self._open(sid)
        return dict.__getitem__(self, sid)

    def get(self, sid, default=None):
        self._open(sid)
        return dict.get(self, sid, default)

    def pop(self, sid, *default):
        self._open(sid)
        return dict.pop(self, sid, *default)

    def setdefault(self, sid, default=None):
        self._open(sid)
        return dict.setdefault(self, sid, default)

    def popitem(self):
        return dict.popitem(self._open_all())

    def values(self):
        return dict.values(self._open_all())

    def items(self):
        return dict.items(self._open_all())

    def __iter__(self):
        return dict.__iter__(self._open_all())

    def copy(self):
        return dict(dict.items(self._open_all()))

    __copy__ = copy

    def __eq__(self, other):
        return dict.__eq__(self._open_all(), other)

    def __ne__(self, other):
        return not self == other

    __hash__ = None

    def __or__(self, other):
        return self.copy() | other

    def __ror__(self, other):
        return other | self.copy()

    def __reduce__(self):
        return (SequenceStates, (self.copy(),))


def _plain(module, cls):
    """A module of exactly this class whose call is the class's own forward."""
    return (type(module) is cls and "forward" not in module.__dict__ and not module._forward_hooks and not module._forward_pre_hooks)


def _is(t, dtype, dev, *shape):
    return t is not None and t.dtype is dtype and t.device == dev and t.shape == shape and t.is_contiguous()


def _sizes(model):
    """(H, P, N, G, taps, d) when every layer can take the step kernels: the published block with bf16 weights, no hooks, equal sizes."""
    emb = model._modules.get("embedding") if _plain(model, Mamba2ForCausalLM) else None
    if emb is None or not _plain(emb, Embedding) or not len(model.layers) or not _plain(model.norm, RMSNorm):
        return None
    if torch_module._global_forward_hooks or torch_module._global_forward_pre_hooks or debug.ENABLED:
        return None
    w = emb.weight
    head = model.head_weight()
    m = model.layers[0].mixer if type(model.layers[0]) is Mamba2Layer else None
    if m is None or not w.is_cuda or w.dtype is not torch.bfloat16 or w.dim() != 2 or not w.is_contiguous():
        return None
    d, bf, f32, dev = w.shape[1], torch.bfloat16, torch.float32, w.device
    if not _is(model.norm.weight, bf, dev, d) or head.dim() != 2 or head.shape[0] < model.config.vocab_size or not _is(head, bf, dev, head.shape[0], d):
        return None
    H, P, N, G, taps = m.nheads, m.headdim, m.d_state, m.ngroups, m.d_conv
    inner, chan = H * P, H * P + 2 * G * N
    # sizes of 8, as the prompt form wants them; a lane of the step kernel owns four neighbouring state columns, two such pieces at most
    if d % 8 or P % 8 or chan % 8 or N % 8 or N > 256 or P > 1024 or not 2 <= taps <= 4 or H % G or inner > 65536:
        return None
    for layer in model.layers:
        sub = layer._modules
        mx = sub.get("mixer")
        if not (_plain(layer, Mamba2Layer) and _plain(mx, Mamba2Block) and _plain(sub["norm"], RMSNorm)):
            return None
        if (mx.nheads, mx.headdim, mx.d_state, mx.ngroups, mx.d_conv, mx.d_inner) != (H, P, N, G, taps, inner):
            return None
        part, own = mx._modules, mx._parameters
        i, o, gn = part["in_proj"], part["out_proj"], part["norm"]
        if not (_plain(i, Linear) and _plain(o, Linear) and _plain(gn, RMSNorm)) or i.bias is not None or o.bias is not None:
            return None
        if not (_is(sub["norm"].weight, bf, dev, d) and _is(i.weight, bf, dev, inner + chan + H, d) and _is(o.weight, bf, dev, d, inner)
                and _is(gn.weight, bf, dev, inner) and _is(own.get("conv_weight"), bf, dev, chan, taps)
                and _is(own.get("conv_bias"), bf, dev, chan) and all(_is(own.get(k), f32, dev, H) for k in ("dt_bias", "A_log", "D"))):
            return None
    return H, P, N, G, taps, d


def _block_of(entry, L, H, P, N, taps, chan, dev):
    """The sequence's block, packed from the per-layer dicts that a prefill or a user left; None when they are not of this form."""
    if isinstance(entry, _Block):
        return entry if entry.ssm.device == dev and entry.ssm.shape == (L, H, P, N) and entry.conv.shape == (2, L, taps - 1, chan) else None
    if not isinstance(entry, list) or len(entry) != L:
        return None
    conv, ssm = [], []
    for layer in entry:
        c, s = layer.get("conv"), layer.get("ssm")
        if (len(layer) != 2 or c is None or s is None or c.dtype is not torch.bfloat16 or s.dtype is not torch.float32 or c.device != dev
                or s.device != dev or c.shape != (1, taps - 1, chan) or s.shape != (1, H, P, N)):
            return None
        conv.append(c)
        ssm.append(s)
    both = torch.empty(2, L, taps - 1, chan, dtype=torch.bfloat16, device=dev)
    torch.cat(conv, out=both[0])
    return _Block(torch.cat(ssm), both)


def decode_step(model, states, seq_ids, last_tokens):
    """Logits [B, vocab] of one token for every sequence, its states advanced; None when model, batch or states are not ones that the
    step kernels take (another device or type, replaced or hooked modules, a sequence twice in the batch, more than 128 rows), in which
    case nothing has changed. Everything is allocated before the first state is written, and a sequence moves on when every kernel has been
    launched; where a launch fails, sequences whose states a kernel may have written are dropped and the others stay as they were."""
    B = len(seq_ids)
    if not (isinstance(states, SequenceStates) and isinstance(model, torch.nn.Module) and 0 < B <= MAX_ROWS and len(last_tokens) == B and len(set(seq_ids)) == B):
        return None
    sizes = _sizes(model)
    if sizes is None or not _lib.available():
        return None
    H, P, N, G, taps, d = sizes
    emb, L = model.embedding.weight, len(model.layers)
    dev, inner, chan = emb.device, H * P, H * P + 2 * G * N
    if dev.index != torch.cuda.current_device():
        return None
    blocks = []
    for sid in seq_ids:
        entry = states.entry(sid)
        if entry is None:
            raise KeyError(sid)
        block = _block_of(entry, L, H, P, N, taps, chan, dev)
        if block is None:
            return None
        blocks.append(block)
    wide = inner + chan + H
    size = L * (taps - 1) * chan * 2
    rows = [int(t) for t in last_tokens]
    for b in blocks:
        base = b.conv.data_ptr()
        rows += [b.ssm.data_ptr(), base + b.cur * size, base + (1 - b.cur) * size]
    table = torch.tensor(rows, dtype=torch.long).to(dev)
    new = lambda *shape: torch.empty(shape, dtype=torch.bfloat16, device=dev)
    x = F.embedding(table[:B], emb)
    res, hn, zx, g, gn, out = new(2, B, d), new(B, d), new(B, wide), new(B, inner), new(B, inner), new(B, d)
    logits = torch.empty(B, model.config.vocab_size, dtype=torch.float32, device=dev)
    a = _lib.SxMambaStepArgs()
    a.hn, a.zx, a.zx_ld, a.g, a.gn, a.out = hn.data_ptr(), zx.data_ptr(), wide, g.data_ptr(), gn.data_ptr(), out.data_ptr()
    a.B, a.d, a.H, a.P, a.N, a.G, a.taps = B, d, H, P, N, G, taps
    a.table, a.status = table.data_ptr() + 8 * B, _lib.status_word(dev).data_ptr()
    half, stream = B * d * 2, _lib.stream()
    try:
        for i, layer in enumerate(model.layers):
            m, own = layer.mixer, layer.mixer._parameters
            # the residual of layer 0 is the embedding, then the two halves of `res` in turn; kernels write only the second of each pair
            a.x = x.data_ptr() if i == 0 else out.data_ptr()
            a.res_in = None if i == 0 else x.data_ptr() if i == 1 else res.data_ptr() + (i & 1) * half
            a.res_out = None if i == 0 else res.data_ptr() + (1 - (i & 1)) * half
            a.layer, a.eps, a.gate_eps = i, layer.norm.eps, m.norm.eps
            a.norm_w, a.gate_norm_w = layer.norm.weight.data_ptr(), m.norm.weight.data_ptr()
            a.in_w, a.out_w = m.in_proj.weight.data_ptr(), m.out_proj.weight.data_ptr()
            a.conv_w, a.conv_b = own["conv_weight"].data_ptr(), own["conv_bias"].data_ptr()
            a.dt_bias, a.a_log, a.D = own["dt_bias"].data_ptr(), own["A_log"].data_ptr(), own["D"].data_ptr()
            _lib.call("sx_mamba2_step", C.byref(a), stream)
        last = x if L == 1 else res[1 - ((L - 1) & 1)]
        _lib.call("sx_rmsnorm_fwd", _lib.ptr(out), _lib.ptr(last), _lib.ptr(model.norm.weight), _lib.ptr(hn), _lib.ptr(None), _lib.ptr(None),
                  _lib.c_ll(B), _lib.c_int(d), _lib.c_float(model.norm.eps), stream)
        gemm(hn, model.head_weight()[:model.config.vocab_size], out=logits)
    except BaseException:
        # kernels may have stepped states where they lie: those sequences are gone rather than half advanced. Lists are never written.
        for sid, b in zip(seq_ids, blocks):
            if dict.get(states, sid) is b:
                dict.pop(states, sid)
        raise
    for sid, b in zip(seq_ids, blocks):
        dict.__setitem__(states, sid, b)
        b.cur = 1 - b.cur
    return logits
