"""Weight-only quantized Linear and the precision plugin that installs it.

Replaces ``lightning.fabric.plugins.BitsandbytesPrecision`` + ``bitsandbytes.nn.Linear4bit`` as used by the
reference (generate/base.py:129-134,151,168; generate/tp.py:127-134,171,190):

* ``QuantPrecision(mode, dtype)`` mirrors ``BitsandbytesPrecision(quantize[4:], dtype)``: ``convert_module`` swaps
  every ``nn.Linear`` (``lm_head`` included) for ``QLinear``; ``module_init_context`` makes ``nn.Linear`` construct
  ``QLinear`` directly (the ``fabric.init_module`` path).
* ``QLinear`` keeps ``weight`` / ``bias`` / ``in_features`` / ``out_features``.  While unquantized it tolerates
  ``linear.weight.data = shard`` and attribute edits (generate/tp.py:37-45); it quantizes ON THE GPU when the module
  is moved to a CUDA device, or when a full-precision ``weight`` arrives through ``load_state_dict`` on a module that
  already lives on CUDA (lit_gpt/utils.py:354-356).  After that ``weight`` is the packed uint8 ``(numel/2, 1)`` tensor
  and ``quant_state`` is the bitsandbytes-0.41 list form ``[absmax, shape, dtype, blocksize, None, quant_type, data_type]``
  (lit_gpt/utils.py:85-87 reads index 1).
* forward: <= 16 activation rows -> the fused dequant-GEMV; more rows (prefill) -> the prefill GEMM.

There is no CPU implementation: calling a QLinear that is not on CUDA raises.
"""
from __future__ import annotations

import contextlib
from typing import Any, Iterator, List, Optional, Set

import torch
import torch.nn as nn
import torch.nn.functional as F

from . import kernels as K
from ._cabi import B200Error

MODES = ("nf4", "nf4-dq", "fp4", "fp4-dq", "int8", "int4")
GEMV_MAX_ROWS = 16


# Captured decode graphs (generate/base.py) bake in the device pointers of the packed / tiled weights: every (re)quantisation
# or packed import anywhere bumps this counter, and the graph cache keys on it.
_WEIGHT_EPOCH = 0


def bump_weight_epoch() -> None:
    global _WEIGHT_EPOCH
    _WEIGHT_EPOCH += 1


def weight_epoch() -> int:
    return _WEIGHT_EPOCH


class QLinear(nn.Module):
    def __init__(self, in_features: int, out_features: int, bias: bool = True, device=None, dtype=None,
                 mode: str = "nf4", compute_dtype: torch.dtype = torch.bfloat16) -> None:
        super().__init__()
        if mode not in MODES:
            raise ValueError(f"unknown quantization mode {mode!r}; expected one of {MODES}")
        self.in_features, self.out_features = in_features, out_features
        self.mode, self.compute_dtype = mode, compute_dtype
        self.quant_type = mode.split("-")[0]  # nf4 | fp4 | int4 | int8
        self.threshold = 6.0  # int8 only: LLM.int8() outlier threshold (Linear8bitLt(threshold=6.0))
        self.SCB: Optional[torch.Tensor] = None  # int8 only: per-row absmax (bitsandbytes Int8Params.SCB); weight holds CB
        self.double_quant = mode.endswith("-dq")  # compress_statistics=True: absmax itself 8-bit quantised
        self.absmax: Optional[torch.Tensor] = None  # fp32 absmax the kernels read (for -dq: the dequantised statistics)
        self.blocksize = 128 if self.quant_type == "int4" else 64
        kw = dict(device=device, dtype=dtype)
        self.weight = nn.Parameter(torch.empty((out_features, in_features), **kw), requires_grad=False)
        self.bias = nn.Parameter(torch.empty(out_features, **kw), requires_grad=False) if bias else None
        self.quant_state: Optional[List[Any]] = None
        # int4 extras (canonical GPTQ-style tensors + the kernel-side interleaved {scale, zero})
        self.scales: Optional[torch.Tensor] = None
        self.qzeros: Optional[torch.Tensor] = None
        self.sz: Optional[torch.Tensor] = None
        # kernel-side tiled copy (csrc/tile.cu) consumed by the streaming GEMV; None when the shape is not covered
        self.tiled: Optional[torch.Tensor] = None
        # row folding of the tiled copy: the flat storage viewed as (out / fold, fold * in) when in_features is not a multiple
        # of the quantisation block (row-parallel shards such as 11008 / 8 = 1376, generate/tp.py:28-45)
        self.fold = 1

    # -- construction from an existing nn.Linear (convert_module path, generate/tp.py:171) -------------------
    @classmethod
    def from_linear(cls, linear: nn.Linear, mode: str, compute_dtype: torch.dtype) -> "QLinear":
        q = cls(linear.in_features, linear.out_features, linear.bias is not None, device="meta", mode=mode,
                compute_dtype=compute_dtype)
        q.weight = nn.Parameter(linear.weight.data, requires_grad=False)
        if linear.bias is not None:
            q.bias = nn.Parameter(linear.bias.data, requires_grad=False)
        if q.weight.is_cuda:
            q.quantize_()
        return q

    @property
    def is_quantized(self) -> bool:
        return self.quant_state is not None

    @property
    def scale(self) -> torch.Tensor:
        """The per-block scale tensor the kernels consume (fp32 absmax, or packed half2 {scale, zero} for int4)."""
        return self.sz if self.quant_type == "int4" else self.absmax

    # -- one resident copy of the weights: the tiled layout is a byte permutation of (weight, scale) ----
    released = False

    def packed(self) -> tuple:
        """(packed weight, scale) in the REFERENCE layout: the stored tensors, or -- after ``release_reference_layout`` -- a
        temporary rebuilt from the tiled copy by ``b200_untile_4bit`` (exact inverse of the tiling, bit for bit)."""
        if not self.released:
            return self.weight.data, self.scale
        N, Kd = self.out_features // self.fold, self.in_features * self.fold
        w, s = K.untile_4bit(self.tiled, N, Kd, self.quant_type, self.blocksize)
        if self.quant_type == "int4":
            return w.view(self.out_features, -1), s.view(self.out_features, -1)
        return w, s

    @torch.no_grad()
    def release_reference_layout(self) -> bool:
        """Drop the reference-layout copy (packed codes + fp32 absmax / fused {scale, zero}) and keep only the tiled one that the
        decode GEMV streams: halves the HBM a 4-bit model occupies (Llama-2-70B int4: 71 -> 36 GB).  Everything that needs the
        reference layout afterwards (prefill GEMM, ``dequantize``, ``state_dict``, checkpoints) rebuilds it on the fly from the
        tiled copy, one Linear at a time.  Returns False (nothing dropped) for modules without a tiled layout."""
        if self.released or not self.is_quantized or self.tiled is None or self.quant_type == "int8":
            return False
        dev = self.weight.device
        self.weight = nn.Parameter(torch.empty(0, dtype=self.weight.dtype, device=dev), requires_grad=False)
        if self.quant_type == "int4":
            self.sz = None
        else:
            self.absmax = None
            if not self.double_quant:
                self.quant_state[0] = None
        self.released = True
        return True

    def _save_to_state_dict(self, destination, prefix, keep_vars):
        super()._save_to_state_dict(destination, prefix, keep_vars)
        if self.released:   # the packed weight as it was before the release
            destination[prefix + "weight"] = self.packed()[0]

    @torch.no_grad()
    def quantize_(self) -> None:
        """Quantize the (CUDA, floating point) weight in place with the library's kernels."""
        if self.is_quantized:
            return
        bump_weight_epoch()
        w = self.weight.data
        if not w.is_cuda:
            raise B200Error("QLinear quantizes on the GPU only (move the module to CUDA); there is no CPU path")
        if w.dtype not in (torch.bfloat16, torch.float16, torch.float32):
            raise B200Error(f"cannot quantize a weight of dtype {w.dtype}")
        # the TP code edits in/out_features and assigns weight.data before the move (generate/tp.py:37-41)
        shape = tuple(w.shape)
        if shape != (self.out_features, self.in_features):
            raise B200Error(f"weight shape {shape} does not match ({self.out_features}, {self.in_features})")
        if self.quant_type == "int8":
            cb, scb = K.quantize_int8(w)
            self.weight = nn.Parameter(cb, requires_grad=False)
            self.SCB = scb
            self.quant_state = [scb, torch.Size(shape), w.dtype, None, None, "int8", None]
            if self.bias is not None and self.bias.dtype != torch.float16:
                self.bias = nn.Parameter(self.bias.data.to(torch.float16), requires_grad=False)
            self.tiled = None
            return
        if self.quant_type == "int4":
            qweight, scales, qzeros, sz = K.quantize_int4(w, self.blocksize)
            self.scales, self.qzeros, self.sz = scales, qzeros, sz
            self.weight = nn.Parameter(qweight, requires_grad=False)
            self.quant_state = [scales, torch.Size(shape), w.dtype, self.blocksize, None, "int4", None]
        else:
            packed, absmax = K.quantize_4bit(w, self.quant_type, self.blocksize)
            self.weight = nn.Parameter(packed, requires_grad=False)
            if self.double_quant:
                # bitsandbytes 0.41 nested form: quant_state[0] = 8-bit absmax, [4] = [offset, [absmax2, code, 256]];
                # the kernels stream the fp32 statistics expanded once here (0.5625 B/param in HBM, 0.5159 on disk)
                qabs, absmax2, offset, absmax = K.double_quant_absmax(absmax)
                self.quant_state = [qabs, torch.Size(shape), w.dtype, self.blocksize, [offset, [absmax2, K.dynamic_map(w.device), 256]],
                                    self.quant_type, None]
            else:
                self.quant_state = [absmax, torch.Size(shape), w.dtype, self.blocksize, None, self.quant_type, None]
            self.absmax = absmax
        if self.bias is not None and self.bias.dtype != self.compute_dtype:
            self.bias = nn.Parameter(self.bias.data.to(self.compute_dtype), requires_grad=False)
        self._build_tiled(shape)

    def _build_tiled(self, shape) -> None:
        """The kernel-side layout: a byte permutation of the packed weight (csrc/tile.cu).  bitsandbytes quantizes the FLAT
        storage, so when in_features is not a multiple of the block the blocks straddle rows; the same flat buffers viewed
        as (N / F, F * K) are block-aligned and tile normally, and the GEMV unfolds the outputs (b200_qgemv_tiled `fold`)."""
        self.tiled, self.fold = None, 1
        N, Kd = int(shape[0]), int(shape[1])
        if K.tiled_bytes(N, Kd, self.quant_type):
            self.tiled = K.tile_4bit(self.weight.data, self.scale, N, Kd, self.quant_type, self.blocksize)
            return
        if self.quant_type != "int4" and Kd % 8 == 0:
            for f in (2, 4):
                if N % f == 0 and K.tiled_bytes(N // f, Kd * f, self.quant_type):
                    self.tiled = K.tile_4bit(self.weight.data, self.scale, N // f, Kd * f, self.quant_type, self.blocksize)
                    self.fold = f
                    return

    # -- pre-quantized checkpoints: the packed tensors go to disk as they are, no re-quantisation on load --
    def export_packed(self) -> dict:
        """CPU copies of exactly what ``quantize_`` produced (packed codes + statistics), keyed for ``import_packed``."""
        if not self.is_quantized:
            raise B200Error("export_packed: the module is not quantized yet")
        pw, ps = self.packed() if self.quant_type != "int8" else (self.weight.data, None)
        out = {"mode": self.mode, "shape": [int(d) for d in self.quant_state[1]], "weight": pw.cpu()}  # plain types: loads with weights_only=True
        if self.quant_type == "int8":
            out["SCB"] = self.SCB.cpu()
        elif self.quant_type == "int4":
            out["scales"], out["qzeros"] = self.scales.cpu(), self.qzeros.cpu()
        elif self.double_quant:
            qs = self.quant_state
            out["qabsmax"], out["offset"], out["absmax2"] = qs[0].cpu(), qs[4][0].cpu() if torch.is_tensor(qs[4][0]) else qs[4][0], qs[4][1][0].cpu()
        else:
            out["absmax"] = ps.cpu()
        if self.bias is not None:
            out["bias"] = self.bias.data.cpu()
        return out

    @torch.no_grad()
    def import_packed(self, st: dict, device: torch.device) -> None:
        """Inverse of ``export_packed`` on ``device``: installs the packed tensors, rebuilds ``quant_state`` and the tiled
        kernel layout (a byte permutation, csrc/tile.cu).  The weights are NOT re-quantized."""
        if st["mode"] != self.mode:
            raise B200Error(f"checkpoint mode {st['mode']!r} does not match module mode {self.mode!r}")
        shape = tuple(st["shape"])
        if shape != (self.out_features, self.in_features):
            raise B200Error(f"packed shape {shape} does not match ({self.out_features}, {self.in_features})")
        dev = torch.device(device)
        if dev.type != "cuda":
            raise B200Error("import_packed: quantized modules live on CUDA only")
        bump_weight_epoch()
        self.weight = nn.Parameter(st["weight"].to(dev), requires_grad=False)
        self.scales = self.qzeros = self.sz = self.tiled = self.absmax = self.SCB = None
        if self.quant_type == "int8":
            self.SCB = st["SCB"].to(dev)
            self.quant_state = [self.SCB, torch.Size(shape), torch.float16, None, None, "int8", None]
        elif self.quant_type == "int4":
            self.scales, self.qzeros = st["scales"].to(dev), st["qzeros"].to(dev)
            self.sz = K.int4_fuse_scale_zero(self.scales, self.qzeros)
            self.quant_state = [self.scales, torch.Size(shape), self.compute_dtype, self.blocksize, None, "int4", None]
        elif self.double_quant:
            qabs, absmax2 = st["qabsmax"].to(dev), st["absmax2"].to(dev)
            offset = st["offset"].to(dev) if torch.is_tensor(st["offset"]) else st["offset"]
            self.absmax = K.dequant_absmax(qabs, absmax2, offset)
            self.quant_state = [qabs, torch.Size(shape), self.compute_dtype, self.blocksize, [offset, [absmax2, K.dynamic_map(dev), 256]], self.quant_type, None]
        else:
            self.absmax = st["absmax"].to(dev)
            self.quant_state = [self.absmax, torch.Size(shape), self.compute_dtype, self.blocksize, None, self.quant_type, None]
        if "bias" in st and self.bias is not None:
            self.bias = nn.Parameter(st["bias"].to(dev), requires_grad=False)
        if self.quant_type != "int8":
            self._build_tiled(shape)

    def dequantize(self, dtype: Optional[torch.dtype] = None) -> torch.Tensor:
        """(out_features, in_features) tensor of code[c] * absmax — bit-exact to oracle/quant_ref.py."""
        if not self.is_quantized:
            raise B200Error("QLinear is not quantized yet")
        dtype = dtype or self.compute_dtype
        shape = self.quant_state[1]
        if self.quant_type == "int8":
            return K.dequantize_int8(self.weight.data, self.SCB, dtype)
        if self.quant_type == "int4":
            return K.dequantize_int4(self.packed()[0], self.scales, self.qzeros, shape[1], self.blocksize, dtype)
        pw, ps = self.packed()
        return K.dequantize_4bit(pw, ps, shape, dtype, self.quant_type, self.blocksize)

    # -- device moves trigger quantization (bitsandbytes: Params4bit.cuda()) --------------------------------
    def _apply(self, fn, recurse: bool = True):
        if self.is_quantized:
            # packed integer tensors must not be cast by .to(dtype); move everything by device only
            probe = fn(torch.empty(0, dtype=torch.float32, device=self.weight.device))
            dev = probe.device
            if dev != self.weight.device:
                if dev.type != "cuda":
                    raise B200Error("a quantized QLinear cannot leave CUDA (no CPU path)")
                self.weight = nn.Parameter(self.weight.data.to(dev), requires_grad=False)
                if self.quant_state[0] is not None:
                    self.quant_state[0] = self.quant_state[0].to(dev)
                if self.double_quant:
                    self.quant_state[4][1][0] = self.quant_state[4][1][0].to(dev)
                    self.quant_state[4][1][1] = self.quant_state[4][1][1].to(dev)
                for name in ("scales", "qzeros", "sz", "tiled", "absmax", "SCB"):
                    t = getattr(self, name)
                    if t is not None:
                        setattr(self, name, t.to(dev))
                if self.bias is not None:
                    self.bias = nn.Parameter(self.bias.data.to(dev), requires_grad=False)
            return self
        super()._apply(fn, recurse)
        if self.weight.is_cuda and self.weight.is_floating_point():
            self.quantize_()
        return self

    # -- full-precision checkpoints load straight into a quantized module (lit_gpt/utils.py:354-356) ---------
    def _load_from_state_dict(self, state_dict, prefix, local_metadata, strict, missing_keys, unexpected_keys, error_msgs):
        wkey, bkey = prefix + "weight", prefix + "bias"
        if wkey in state_dict and state_dict[wkey].is_floating_point():
            w = state_dict[wkey]
            if tuple(w.shape) != (self.out_features, self.in_features):
                error_msgs.append(f"size mismatch for {wkey}: checkpoint {tuple(w.shape)} vs module "
                                  f"({self.out_features}, {self.in_features})")
                return
            target = self.weight.device
            self.quant_state, self.scales, self.qzeros, self.sz, self.tiled, self.absmax, self.SCB = None, None, None, None, None, None, None
            if target.type == "cuda":
                self.weight = nn.Parameter(w.detach().to(target), requires_grad=False)
                self.quantize_()
            else:  # meta / cpu: keep the full-precision weight; quantization happens at the device move
                self.weight = nn.Parameter(w.detach(), requires_grad=False)
            if self.bias is not None:
                if bkey in state_dict:
                    b = state_dict[bkey].detach()
                    self.bias = nn.Parameter(b.to(target) if target.type == "cuda" else b, requires_grad=False)
                elif strict:
                    missing_keys.append(bkey)
            elif bkey in state_dict and strict:
                unexpected_keys.append(bkey)
            return
        super()._load_from_state_dict(state_dict, prefix, local_metadata, strict, missing_keys, unexpected_keys, error_msgs)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        if not self.is_quantized or not x.is_cuda:
            raise B200Error("QLinear.forward needs the module quantized on CUDA and a CUDA input; there is no CPU "
                            "fallback (move the model with fabric.setup_module / .to('cuda'))")
        in_dtype = x.dtype
        if self.quant_type == "int8":  # LLM.int8() computes in fp16 (bitsandbytes casts other dtypes to fp16 too)
            try:
                y = K.linear_int8(x if in_dtype == torch.float16 else x.to(torch.float16), self.weight.data, self.SCB, self.bias, self.threshold)
            except NotImplementedError:  # in_features not a multiple of 64 (toy configs): dequantised fp16 product
                y = F.linear(x.to(torch.float16), self.dequantize(torch.float16), self.bias)
            return y if in_dtype == torch.float16 else y.to(in_dtype)
        if in_dtype != torch.bfloat16:
            x = x.to(torch.bfloat16)
        rows = x.numel() // self.in_features
        if torch.compiler.is_compiling():  # traced: one opaque b200gpt::qlinear* node (lit_gpt_b200/ops.py), no graph break
            from . import ops  # noqa: F401

            if self.fold == 1 and self.streams(rows):
                y = torch.ops.b200gpt.qlinear_tiled(x, self.tiled, self.out_features, self.in_features, self.quant_type, self.blocksize, self.bias)
            else:
                pw, ps = self.packed()
                y = torch.ops.b200gpt.qlinear(x, pw, ps, self.out_features, self.in_features, self.quant_type,
                                              self.blocksize, self.bias)
            return y if in_dtype == torch.bfloat16 else y.to(in_dtype)
        # <= 16 rows: the streaming GEMV, provided the activation rows fit its shared-memory plan (a 16-token prompt at
        # K = 8192 does not: that call is a small prefill and takes the GEMM); shapes without a tiled layout (toy
        # configs) keep the reference-layout GEMV
        if rows <= GEMV_MAX_ROWS and (self.tiled is None or self.streams(rows)):
            bias = self.bias
            if self.tiled is not None and (self.fold == 1 or bias is None):
                y = K.qgemv_tiled_rows(x, self.tiled, self.out_features, self.in_features, self.quant_type, self.blocksize, bias, self.fold)
            else:
                y = self.gemv(x, bias=bias)
        else:
            y = prefill_linear(self, x)
        return y if in_dtype == torch.bfloat16 else y.to(in_dtype)

    def streams(self, rows: int, swiglu: bool = False) -> bool:
        """True when `rows` activation rows run on the streaming GEMV over the tiled layout (asked of the library: the
        kernel's shared-memory plan must hold the activation rows)."""
        return (self.tiled is not None and rows <= GEMV_MAX_ROWS
                and K.qgemv_tiled_supported(self.out_features, self.in_features, self.quant_type, rows, swiglu, self.fold))

    def gemv(self, x: torch.Tensor, other: Optional["QLinear"] = None, prefetch: Optional[torch.Tensor] = None,
             **kw: Any) -> torch.Tensor:
        """<= 16 activation rows through the fused dequant-GEMV: the streaming kernel over the tiled layout when the
        shape is covered (and the activation fits its shared memory), else the reference-layout kernel.
        ``other``: the up-projection for the fused SwiGLU pair (this module being the gate)."""
        if self.quant_type == "int8":
            raise B200Error("QLinear.gemv is the 4-bit fused path; int8 modules go through forward()")
        rows = x.numel() // self.in_features
        plain = not any(kw.get(k) is not None for k in ("norm_weight", "delta", "x_out", "bias", "bias2"))
        if (other is None or (other.tiled is not None and other.fold == 1 and self.fold == 1)) and (self.fold == 1 or plain) \
                and self.streams(rows, swiglu=other is not None):
            return K.qgemv_tiled(x, self.tiled, self.out_features, self.in_features, self.quant_type, self.blocksize,
                                 tiled2=None if other is None else other.tiled, prefetch=prefetch, fold=self.fold, **kw)
        if other is not None:
            ow, os_ = other.packed()
            kw.update(packed2=ow, scale2=os_)
        kw.pop("bias2", None)
        kw.pop("kv_hint", None)
        if kw.pop("attn", None) is not None:
            raise B200Error("QLinear.gemv: the fused attention step needs the streaming kernel (ask K.qgemv_attn_fusable first)")
        pw, ps = self.packed()
        return K.qgemv(x, pw, ps, self.out_features, self.in_features, self.quant_type,
                       self.blocksize, **kw)

    def extra_repr(self) -> str:
        return f"in_features={self.in_features}, out_features={self.out_features}, bias={self.bias is not None}, mode={self.mode}"


def prefill_linear(q: QLinear, x: torch.Tensor) -> torch.Tensor:
    """T > 16 rows: the tcgen05 / TMEM dequant-GEMM: weights are dequantised tile by tile, in tensor memory (csrc/qgemm_short.cu,
    most calls of up to 256 rows) or in shared memory (csrc/qgemm.cu), the bf16 matrix never exists in HBM.  Shapes it does not cover (K not a multiple of the quantisation
    block, N % 8 != 0: toy configs only) take the reference's own formulation -- dequantize_4bit to bf16, then a
    library GEMM -- with the dequantisation done by this library's kernel."""
    if x.dtype == torch.bfloat16:
        try:
            pw, ps = q.packed()
            return K.qgemm(x, pw, ps, q.out_features, q.in_features, q.quant_type, q.blocksize, bias=q.bias)
        except NotImplementedError:
            pass
    w = q.dequantize(torch.bfloat16)
    return F.linear(x, w, q.bias)


def _called_plainly(m: nn.Module) -> bool:
    """True when calling `m` does nothing but run QLinear.forward: no override of it, no hook on the module or on all modules."""
    every = torch.nn.modules.module
    return (type(m).forward is QLinear.forward and type(m).__call__ is nn.Module.__call__ and "forward" not in m.__dict__
            and not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks or every._global_forward_hooks
                     or every._global_forward_pre_hooks or every._global_backward_hooks or every._global_backward_pre_hooks))


def _plain_pair(gate: nn.Module, up: nn.Module) -> bool:
    """Plain 4-bit modules of one layout without a bias or a hook (a hook wants the projections' own outputs) whose reference layouts are resident."""
    if not all(isinstance(m, QLinear) and _called_plainly(m) and m.is_quantized and not m.released and m.quant_type != "int8" and m.bias is None
               for m in (gate, up)):
        return False
    return (gate.quant_type == up.quant_type and gate.blocksize == up.blocksize and gate.in_features == up.in_features
            and gate.out_features == up.out_features)


def prefill_pair(gate: nn.Module, up: nn.Module, rows: int) -> bool:
    """True where the two projections of a gated MLP can be one launch with the product in its epilogue, at sizes the library calls the shorter way."""
    return _plain_pair(gate, up) and K.qgemm_swiglu_supported(rows, gate.out_features, gate.in_features, gate.quant_type, gate.blocksize)


def short_pair(gate: nn.Module, up: nn.Module, rows: int) -> bool:
    """``prefill_pair`` for what else the library does in one launch: up to 208 rows, and beyond 512 where ``prefill_pair`` says no.  Up to 208 rows that launch copies
    scales 16 bytes at a time: those that begin elsewhere (views into a larger buffer) are left to the other launches, which read them one by one."""
    return (_plain_pair(gate, up) and K.qgemm_pair_workspace(rows, gate.out_features, gate.in_features, gate.quant_type, gate.blocksize) >= 0
            and (rows > 208 or all(m.packed()[1].data_ptr() % 16 == 0 for m in (gate, up))))


class QuantPrecision:
    """Mirror of ``lightning.fabric.plugins.BitsandbytesPrecision(mode, dtype, ignore_modules)``."""

    precision = "quantized"

    def __init__(self, mode: str, dtype: Optional[torch.dtype] = None, ignore_modules: Optional[Set[str]] = None) -> None:
        if mode.startswith(("bnb.", "gptq.")):
            mode = mode.split(".", 1)[1]
        if mode not in MODES:
            raise ValueError(f"Unsupported quantization mode {mode!r}; supported: {MODES}")
        self.mode = mode
        self.dtype = dtype or (torch.float16 if mode == "int8" else torch.bfloat16)
        if mode == "int8":
            # tutorials/quantize.md:111: bnb.int8 runs with --precision 16-true; bf16 activations are cast per call
            if self.dtype not in (torch.float16, torch.bfloat16):
                raise NotImplementedError(f"bnb.int8 computes in fp16 (requested {self.dtype}); use --precision 16-true")
        elif self.dtype != torch.bfloat16:
            raise NotImplementedError(f"b200gpt computes in bf16 (requested {self.dtype}); use --precision bf16-true")
        self.ignore_modules = set(ignore_modules or ())

    def convert_module(self, module: nn.Module) -> nn.Module:
        n = _convert_layers(module, self.mode, self.dtype, self.ignore_modules)
        if n == 0 and not any(isinstance(m, QLinear) for m in module.modules()):
            raise TypeError("You are using the quantization plugin, but your model has no Linear layers.")
        for m in module.modules():  # everything that is not a packed weight computes in `dtype`
            for name, p in list(m.named_parameters(recurse=False)):
                if p.is_floating_point() and p.dtype != self.dtype and not isinstance(m, QLinear):
                    setattr(m, name, nn.Parameter(p.data.to(self.dtype), requires_grad=False))
        return module

    @contextlib.contextmanager
    def tensor_init_context(self) -> Iterator[None]:
        prev = torch.get_default_dtype()
        torch.set_default_dtype(self.dtype)
        try:
            yield
        finally:
            torch.set_default_dtype(prev)

    @contextlib.contextmanager
    def module_init_context(self) -> Iterator[None]:
        """Default dtype + ``torch.nn.Linear`` constructs QLinear (the reference's fabric.init_module path)."""
        mode, dtype = self.mode, self.dtype
        orig = torch.nn.Linear

        class _Bound(QLinear):
            def __init__(self, in_features, out_features, bias=True, device=None, dtype_=None, **kw):
                super().__init__(in_features, out_features, bias, device=device, dtype=dtype_, mode=mode, compute_dtype=dtype)

        with self.tensor_init_context():
            torch.nn.Linear = _Bound  # type: ignore[misc]
            try:
                yield
            finally:
                torch.nn.Linear = orig  # type: ignore[misc]

    forward_context = tensor_init_context


def _convert_layers(module: nn.Module, mode: str, dtype: torch.dtype, ignore: Set[str], prefix: str = "") -> int:
    n = 0
    for name, child in module.named_children():
        full = f"{prefix}.{name}" if prefix else name
        if isinstance(child, nn.Linear) and not any(full.startswith(i) for i in ignore):
            setattr(module, name, QLinear.from_linear(child, mode, dtype))
            n += 1
        else:
            n += _convert_layers(child, mode, dtype, ignore, full)
    return n
