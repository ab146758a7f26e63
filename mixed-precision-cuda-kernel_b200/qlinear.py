"""Packed inference CherryQ linear (reference: llama/qlinear.py:13-199).

Same constructor, buffers (`cherry_indices` int16 (C,), `cherry_weight` fp16 (C, N),
`qweight` uint8 (K'/8*bits, N), `scales` fp16 (ceil(K'/G), N), optional `bias`),
`pack()`, `unpack()`, `forward()` and class-level `dmode()` switch as the reference,
so a state dict written by the reference loads into it.  What runs underneath is
different: pack and unpack are GPU kernels, and forward runs on re-packed copies of
the buffers that the module owns (made on first use of the kernel family that needs
them; `release_reference_buffers()` drops the originals afterwards):
  decode batches        row-tile layout, the row kernel, up to RowLayer.row_limit rows
  larger batches        tile layout, the tensor-core GEMM
  layers the row kernel does not take: stream layout, the stream matvec, below 8 rows
The kernel of a call depends on the layer and the number of rows only, never on the calls before it.
All of it needs a CUDA device.
"""
import math
from contextlib import contextmanager

import torch
import torch.nn as nn

from . import load_quant_cuda


GEMM_MIN_ROWS = 8       # layers the row kernel does not take: the stream matvec below, the tensor-core GEMM from here on


class QuantLinear(nn.Module):
    _layerwise_dequantize = True

    @classmethod
    @contextmanager
    def dmode(cls, layerwise_dequantize=True):
        mode = cls._layerwise_dequantize
        cls._layerwise_dequantize = layerwise_dequantize
        try:
            yield
        finally:
            cls._layerwise_dequantize = mode

    def __init__(self, w_bits, group_size, quantizer, cherry_fraction: float, in_features, out_features,
                 bias=True, **kwargs):
        super().__init__()
        self.in_features = in_features
        self.out_features = out_features
        self.w_bits = w_bits
        self.group_size = group_size if group_size != -1 else in_features
        self.quantizer = quantizer
        self.cherry_fraction = cherry_fraction
        self.num_cherries = math.ceil(in_features * cherry_fraction) // 8 * 8
        self.num_normal = self.in_features - self.num_cherries
        assert in_features % 8 == 0
        assert out_features % 8 == 0
        self.register_buffer("cherry_indices", torch.zeros(self.num_cherries, dtype=torch.int16))
        self.register_buffer("cherry_weight", torch.zeros((self.num_cherries, out_features), dtype=torch.float16))
        self.register_buffer("qweight", torch.zeros((self.num_normal // 8 * w_bits, out_features), dtype=torch.uint8))
        self.register_buffer("scales", torch.zeros((math.ceil(self.num_normal / self.group_size), out_features),
                                                   dtype=torch.float16))
        if bias:
            self.register_buffer("bias", torch.zeros(out_features, dtype=torch.float16))
        else:
            self.bias = None
        self.dequantized = False
        self._prepared = None        # stream layout (PreparedLayer)
        self._row = None             # row-tile layout (RowLayer)
        self._tile = None            # tile layout of the GEMM (TileLayer)
        self._fast = None            # PackedForward over the copies made so far
        self._row_rows = None        # rows the row kernel serves, 0 = none, None = not asked yet
        self._prepared_key = None    # BufferGuard of the buffers the copies were made from, or "released"

    # ------------------------------------------------------------------ pack / unpack
    @torch.inference_mode()
    def pack(self, linear):
        """GPU version of llama/qlinear.py:67-118; `linear` is the training-side layer."""
        qc = load_quant_cuda()
        if linear.bias is not None:
            self.bias = linear.bias.half()
        weight = linear.weight.detach()
        if not weight.is_cuda:
            if not torch.cuda.is_available():
                raise RuntimeError("QuantLinear.pack needs a CUDA device (there is no CPU path)")
            weight = weight.cuda()
        weight = weight.contiguous()
        if weight.dtype not in (torch.float16, torch.float32):
            weight = weight.float()
        idx = linear.cherry_indices.to(device=weight.device, dtype=torch.int32).contiguous()
        gs = linear.group_size if linear.group_size != -1 else self.in_features
        q, s, cw, ci = qc.pack(weight, idx, self.w_bits, gs)
        self.qweight, self.scales, self.cherry_weight, self.cherry_indices = q, s, cw, ci
        self._drop_copies()

    @torch.inference_mode()
    def unpack(self):
        """GPU version of llama/qlinear.py:120-162: dense (out, in) fp16 weight."""
        qc = load_quant_cuda()
        self._require_cuda()
        return qc.unpack_dense(self.qweight, self.scales, self.cherry_weight, self.cherry_indices,
                               self.w_bits, self.in_features, self.group_size)

    # ------------------------------------------------------------------ forward
    def _require_cuda(self):
        if not self.qweight.is_cuda:
            raise RuntimeError("QuantLinear buffers must be on a CUDA device (there is no CPU path)")

    def _buffer_key(self):
        """The record of the reference buffers as they are now (storages, addresses, versions)."""
        return load_quant_cuda().BufferGuard(self.qweight, self.scales, self.cherry_weight, self.cherry_indices)

    def _drop_copies(self):
        self._prepared = None
        self._row = None
        self._tile = None
        self._fast = None
        self._row_rows = None
        self._prepared_key = None

    def __getstate__(self):
        """For copy and pickle: without the re-packed copies, which the other module makes again on first use.  (After a
        release they are all there is of the weights, and cannot be pickled: restore the reference buffers first.)"""
        state = self.__dict__.copy()
        if self._prepared_key != "released":
            state.update(_prepared=None, _row=None, _tile=None, _fast=None, _row_rows=None, _prepared_key=None)
        return state

    def _sync_key(self):
        """Forgets the re-packed copies when the reference buffers were replaced or written to."""
        if self._prepared_key == "released":
            return
        bufs = (self.qweight, self.scales, self.cherry_weight, self.cherry_indices)
        if self._prepared_key is None or not self._prepared_key.holds(*bufs):
            self._drop_copies()
            self._prepared_key = self._buffer_key()

    def _source_buffers(self):
        """The four reference buffers: the module's own, or rebuilt from a copy after a release."""
        if self._prepared_key != "released":
            return self.qweight, self.scales, self.cherry_weight, self.cherry_indices
        src = self._row if self._row is not None else self._prepared
        return src.unprepare()

    def prepared(self):
        """The stream-layout copy of this layer (built on first use)."""
        self._sync_key()
        if self._prepared is None:
            qc = load_quant_cuda()
            self._require_cuda()
            q, s, cw, ci = self._source_buffers()
            self._prepared = qc.PreparedLayer(q, s, cw, ci, self.w_bits, self.in_features, self.group_size)
        return self._prepared

    def _row_limit(self):
        """Rows up to which the row kernel serves this layer, 0 where it does not take it."""
        self._sync_key()
        if self._row_rows is None:
            qc = load_quant_cuda()
            self._require_cuda()
            self._row_rows = qc.RowLayer.row_limit(self.w_bits, self.in_features, self.out_features, self.num_cherries,
                                                   self.group_size)
        return self._row_rows

    def row_layer(self, rows=1):
        """The row-tile copy for the decode kernel (built on first use), or None where the kernel does not take the layer
        or that many rows."""
        if rows > self._row_limit():
            return None
        if self._row is None:
            qc = load_quant_cuda()
            q, s, cw, ci = self._source_buffers()
            self._row = qc.RowLayer(q, s, cw, ci, self.w_bits, self.in_features, self.group_size)
            self._fast = None
        return self._row

    @torch.inference_mode()
    def forward_swiglu(self, gate: torch.Tensor, up: torch.Tensor):
        """This layer applied to silu(gate) * up (the down projection of the reference's LlamaMLP.forward,
        llama/modeling_llama_quant.py): for decode batches the product is formed while the kernel stages its
        input (no separate element-wise kernel, no intermediate tensor): the result is that of
        forward(silu_mul(gate, up)), with the fast exponential.  Other cases compute the product first, with the
        values of the torch expression, silu in fp32."""
        rows = gate.numel() // gate.shape[-1]
        row = self.row_layer(rows) if (self._layerwise_dequantize and self.w_bits in (3, 4)
                                       and gate.dtype == torch.float16) else None
        if row is None:
            if gate.is_cuda and gate.dtype == up.dtype == torch.float16 and gate.shape == up.shape and gate.numel():
                return self(load_quant_cuda().silu_mul(gate.contiguous(), up.contiguous(), True))
            return self(nn.functional.silu(gate.float()).to(gate.dtype) * up)
        g2 = gate.reshape(rows, gate.shape[-1]).contiguous()
        u2 = up.reshape(rows, up.shape[-1]).contiguous()
        out = torch.empty(rows, self.out_features, dtype=torch.float16, device=g2.device)
        row.matvec_swiglu(g2, u2, out)
        out = out.reshape(gate.shape[:-1] + (self.out_features,))
        if self.bias is not None:
            out += self.bias
        return out

    def release_reference_buffers(self):
        """Keeps only the re-packed copies (roughly halves the weight memory);
        `restore_reference_buffers` rebuilds the four buffers bit-exactly."""
        if self.row_layer() is None:
            self.prepared()
        dev = self.qweight.device
        for name in ("qweight", "scales", "cherry_weight", "cherry_indices"):
            setattr(self, name, torch.empty(0, dtype=getattr(self, name).dtype, device=dev))
        self._prepared_key = "released"
        self._fast = None

    def restore_reference_buffers(self):
        q, s, cw, ci = self._source_buffers()
        self.qweight, self.scales, self.cherry_weight, self.cherry_indices = q, s, cw, ci
        self._prepared_key = self._buffer_key()
        self._fast = None

    def tile_layer(self):
        """The tile-layout copy of the tensor-core GEMM (built on first use)."""
        self._sync_key()
        if self._tile is None:
            qc = load_quant_cuda()
            self._require_cuda()
            q, s, cw, ci = self._source_buffers()
            self._tile = qc.TileLayer(q, s, cw, ci, self.w_bits, self.in_features, self.group_size)
            self._fast = None
        return self._tile

    def forward(self, x: torch.Tensor):
        if self._fast is not None and self._layerwise_dequantize:
            out = self._fast(x, self._buffers, self.bias)
            if out is not None:
                return out
        return self._forward(x)

    @torch.inference_mode()
    def _forward(self, x: torch.Tensor):
        if self._layerwise_dequantize:
            if self.w_bits not in (3, 4):
                raise NotImplementedError(f"{self.w_bits} bit kernel is not implemented yet.")
            out_shape = x.shape[:-1] + (self.out_features,)
            x2 = x.reshape(-1, x.shape[-1])
            if x2.dtype != torch.float16:
                x2 = x2.half()
            x2 = x2.contiguous()
            rows = x2.shape[0]
            limit = self._row_limit()
            gemm_rows = limit + 1 if limit else GEMM_MIN_ROWS
            out = torch.empty(rows, self.out_features, dtype=torch.float16, device=x2.device)
            if rows <= limit:
                self.row_layer().matvec(x2, out, False)
            elif rows < gemm_rows:
                self.prepared().matvec(x2, out, False)
            elif self.w_bits == 4 and self.group_size < 128 and self._prepared_key != "released":
                raise RuntimeError("4-bit layers with groups narrower than 128 have no kernel for large batches")
            else:
                # more rows: the tensor-core GEMM on this module's tile-layout copy
                self.tile_layer().gemm(x2, out, False)
            if self._fast is None and (self._row is not None or self._tile is not None):
                guard = None if self._prepared_key == "released" else self._prepared_key
                self._fast = load_quant_cuda().PackedForward(self._row, self._tile, guard, limit, gemm_rows)
            out = out.reshape(out_shape).to(x.dtype)
        else:
            if not self.dequantized:
                self.qweight = self.unpack()
                del self.cherry_indices
                del self.cherry_weight
                del self.scales
                self._drop_copies()
                torch.cuda.empty_cache()
                self.dequantized = True
            out = nn.functional.linear(x, self.qweight)
        if self.bias is not None:
            out += self.bias
        return out


def _alike(layers):
    """Whether one launch can serve these layers, by their sizes."""
    first = layers[0]
    same = all((l.w_bits, l.in_features, l.num_cherries, l.group_size) ==
               (first.w_bits, first.in_features, first.num_cherries, first.group_size) for l in layers)
    return 1 < len(layers) <= 4 and same and QuantLinear._layerwise_dequantize and first.w_bits in (3, 4)


def _row_copies(layers, rows):
    """The row-tile copies of layers that one launch of the row kernel can serve for that many rows, or None."""
    if not _alike(layers):
        return None
    rls = []
    for l in layers:
        r = l.row_layer(rows)
        if r is None:
            return None
        rls.append(r)
    return rls


# Rows up to which the GEMM serves layers together: one token block of 32.  Microseconds one after another and together, 16
# and 32 rows: 8192 -> (8192, 1024, 1024) 47 and 34, 53 and 39; 8192 -> 2 x 28672 97 and 90, 97 and 90; 5120 -> 3 x 5120 46 and
# 36, 54 and 46; 4096 -> 3 x 4096 40 and 34, 47 and 44.  Beyond, storing the layers' parts in one launch costs more than
# the launches: 64 rows 4096 -> 3 x 4096 61 and 65, 128 rows 5120 -> 3 x 5120 86 and 95, 512 rows 162 and 179.
GEMM_TOGETHER_ROWS = 32


# what a call runs, as defined here and in torch (a replaced method of the class is not the same object)
_OWN_METHODS = {name: getattr(QuantLinear, name) for name in ("__call__", "forward", "_forward")}


def _calls_only_forward(layer):
    """Whether layer(x) is QuantLinear.forward and nothing else: no hook on the module or on all modules, no method replaced on
    the instance (as device-placement wrappers and adapters do) or its class, not compiled."""
    hooked = layer._forward_hooks or layer._forward_pre_hooks or layer._backward_hooks or layer._backward_pre_hooks
    if hooked or nn.modules.module._has_any_global_hook() or layer._compiled_call_impl is not None:
        return False
    return all(getattr(type(layer), name) is own and name not in layer.__dict__ for name, own in _OWN_METHODS.items())


def _tile_copies(layers, x, rows):
    """The tile-layout copies of layers whose own forward of `x` is the GEMM on them and nothing else, or None."""
    first = layers[0]
    if not (rows <= GEMM_TOGETHER_ROWS and _alike(layers) and x.is_cuda and x.dtype == torch.float16 and x.shape[-1] == first.in_features
            and (first.w_bits == 3 or first.group_size >= 128)):
        return None
    # One look at the buffers of each layer (four attributes of a module, their storages and versions): with one for each question
    # a call of three layers took the host 46 us, 33 like this; their own three calls 40.
    tls = []
    for l in layers:
        if not _calls_only_forward(l):
            return None
        limit = l._row_limit()
        if rows < (limit + 1 if limit else GEMM_MIN_ROWS):
            return None
        tile = l._tile
        tls.append(tile if tile is not None else l.tile_layer())
    return tls


@torch.inference_mode()
def _gemm_together(layers, tls, x, rows):
    outs = load_quant_cuda().tile_layers_gemm(tls, x.reshape(rows, x.shape[-1]).contiguous())
    outs = [o.reshape(x.shape[:-1] + (l.out_features,)) for l, o in zip(layers, outs)]
    for l, o in zip(layers, outs):
        if l.bias is not None:
            o += l.bias
    return outs


def _row_outputs(layers, shape, dtype, rows, device, launch):
    """Outputs of `layers` as views of one buffer, filled by launch(outs)."""
    widths = [l.out_features for l in layers]
    buf = torch.empty(rows, sum(widths), dtype=torch.float16, device=device)
    outs = list(buf.split(widths, dim=1))                       # views of one buffer: one row stride
    launch(outs)
    res = []
    for l, o in zip(layers, outs):
        o = o.contiguous().reshape(shape[:-1] + (l.out_features,)).to(dtype)
        if l.bias is not None:
            o += l.bias
        res.append(o)
    return res


def forward_shared_input(layers, x: torch.Tensor):
    """Outputs of several packed layers applied to the same input (q / k / v, gate / up of the
    reference's LLaMA, llama/modeling_llama_quant.py): for layers that agree in bits, in_features, cherry
    count and group size this is ONE launch of the row-tile kernel per four rows of a decode batch (up to the
    layers' row limit), with the SMs divided among the layers, and ONE launch of the GEMM for batches beyond, up
    to 32 rows; every other case is the layers' own forward, one by one.  The results are bit-identical to the separate calls."""
    layers = list(layers)
    rows = x.numel() // x.shape[-1]
    rls = _row_copies(layers, rows)
    if rls is None:
        tls = _tile_copies(layers, x, rows)
        return [l(x) for l in layers] if tls is None else _gemm_together(layers, tls, x, rows)
    x2 = x.reshape(rows, x.shape[-1])
    if x2.dtype != torch.float16:
        x2 = x2.half()
    x2 = x2.contiguous()
    return _row_outputs(layers, x.shape, x.dtype, rows, x2.device,
                        lambda outs: load_quant_cuda().row_layers_matvec(rls, x2, outs, False))


def forward_normed_input(layers, h: torch.Tensor, delta, weight: torch.Tensor, eps: float):
    """(outputs, h + delta): the layers applied to the RMS norm of h + delta (delta may be None), the residual stream of the
    reference's decoder layer (llama/modeling_llama_quant.py:724-785).  One fp16 row: the norm rides in the
    launch of forward_shared_input; everything else is the norm kernel and that function.

    Every CTA reads the whole rows twice, row after row, so the launch saved pays for one row only.  Microseconds with the norm
    inside and in front, one and two rows: 4096 -> 3 x 4096 8.0 and 9.3, 21.5 and 19.3; 8192 -> (8192, 1024, 1024) 12.1 and 13.1,
    27.0 and 25.1; 16384 -> 2 x 4096 18.0 and 18.7, 31.0 and 28.0; four rows 25.6 and 23.0, 34.3 and 29.7, 40.3 and 32.5."""
    layers = list(layers)
    qc = load_quant_cuda()
    rows = h.numel() // h.shape[-1]
    plain = all(t is None or (t.dtype == torch.float16 and t.is_contiguous() and t.data_ptr() % 16 == 0) for t in (h, delta, weight))
    rls = _row_copies(layers, rows) if rows == 1 and plain and h.dim() == 2 else None
    if rls is None:
        if delta is None:
            return forward_shared_input(layers, qc.rmsnorm(h, None, weight, eps, False)[0]), h
        y, h = qc.rmsnorm(h, delta, weight, eps, True)
        return forward_shared_input(layers, y), h
    sums = []
    outs = _row_outputs(layers, h.shape, h.dtype, rows, h.device,
                        lambda o: sums.append(qc.row_layers_matvec_norm(rls, h, delta, weight, eps, o)))
    return outs, sums[0]
