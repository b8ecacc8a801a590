"""``QuantLinear`` -- the module that ``make_quant(..., use_tvm=True)`` installs.

Mirrors the constructor / ``pack`` / ``forward`` surface of the reference's TVM
module (``auto_gptq/nn_modules/qlinear_tvm.py:10-158``) but keeps the standard
AutoGPTQ buffers of ``auto_gptq/nn_modules/qlinear.py:40-59`` (``qweight``,
``qzeros``, ``scales``, ``g_idx``, ``bias``), so ordinary GPTQ checkpoints load
unchanged.  ``forward`` runs on the GPU only: up to 16 rows (8 where groups cut
32-row blocks) go to the decode GEMV, more rows to the tcgen05 dequant-GEMM.  There is no M padding, no per-shape
kernel cache and no tuner (the reference's ``tvm_untils/cache.py`` and
``pycuda_warpper.py`` have no counterpart here).
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn as nn

from . import _lib, ops

_buffer_hooks = nn.modules.module._global_buffer_registration_hooks
GEMV_MAX_M = 8
GEMV_WIDE_M = 16    # the streaming kernel takes up to 16 rows (a plan of 9..16 rows: b200gptq_gemv_plan_create)


def _pack_fields(vals: torch.Tensor, bits: int) -> torch.Tensor:
    """Pack ``vals`` (int64 ``[R, C]``, R % 32 == 0) along dim 0 into int32 words.

    2/4/8 bits: field j of a word at bit ``bits*j``.  3 bits: 32 fields form a
    96-bit little-endian stream over three words.  Over-wide values spill into
    the neighbouring fields exactly like the reference's un-masked ``|=``
    (qlinear.py:111-134).
    """
    R, C = vals.shape
    if bits in (2, 4, 8):
        pf = 32 // bits
        v = vals.reshape(R // pf, pf, C)
        shifts = (torch.arange(pf, dtype=torch.int64) * bits).reshape(1, pf, 1)
        words = torch.zeros((R // pf, C), dtype=torch.int64)
        for j in range(pf):
            words |= (v[:, j] << (bits * j)) & 0xFFFFFFFF
        del shifts
    else:
        v = vals.reshape(R // 32, 32, C)
        words = torch.zeros((R // 32, 3, C), dtype=torch.int64)
        for j in range(32):
            bit = 3 * j
            wi, sh = bit // 32, bit % 32
            words[:, wi] |= (v[:, j] << sh) & 0xFFFFFFFF
            if sh > 29:  # the field straddles into the next word
                mask = (1 << (sh + 3 - 32)) - 1
                words[:, wi + 1] |= (v[:, j] >> (32 - sh)) & mask
        words = words.reshape(R // 32 * 3, C)
    words = torch.where(words >= 2**31, words - 2**32, words)
    return words.to(torch.int32)


def row_rules(K: int, groupsize: int, has_g_idx: bool, uniform: bool):
    """``(gemm_ok, gemv_rows)`` of a run-time layout: whether the tensor-core kernel takes it (one group per aligned 32-row
    block; ``uniform`` says so of a ``g_idx``), and the largest batch that goes through the GEMV in one pass.

    9 to 16 rows: one pass of the streaming GEMV, where it takes the layer, beats the tensor-core kernel's 16-row tile, whose
    weight warps are the bottleneck (9216 x 9216, 3 bits: 21 against 40 us; 4096 x 4096, 4 bits: 7.9 against 16.6).  The kernel for
    pairs of SMs has not been set against it (it takes 19.9 us for 32 rows of 9216 x 9216).  It is also where results change by a rounding: the GEMM multiplies the reference's fp16 ``scale * (q - zero)``, the GEMV the exact field
    and the scale in fp32 (2.1e-4 against 2.8e-4 from the exact product)."""
    whole_blocks = groupsize % 32 == 0
    gemm_ok = uniform if has_g_idx else whole_blocks
    streams = not has_g_idx and (whole_blocks or groupsize >= K)
    return gemm_ok, GEMV_WIDE_M if streams else GEMV_MAX_M


def _version(t) -> int:
    """Counts what is written in place to a tensor (tensors of inference mode do not count)."""
    return 0 if t.is_inference() else t._version


def _same(a, b) -> bool:
    """Of two results of ``QuantLinear._constants``: the same tensors, at the same addresses, with the same numbers in them."""
    return a[0] is b[0] and a[1] is b[1] and a[2] is b[2] and a[3:] == b[3:]


class QuantLinear(nn.Module):
    def __init__(self, bits, groupsize, infeatures, outfeatures, bias):
        super().__init__()
        if bits not in [2, 3, 4, 8]:
            raise NotImplementedError("Only 2,3,4,8 bits are supported.")
        if infeatures % 32 != 0 or outfeatures % 32 != 0:
            raise ValueError("infeatures and outfeatures must be multiples of 32 (the packed format needs it)")
        self.infeatures = infeatures
        self.outfeatures = outfeatures
        self.bits = bits
        self.groupsize = groupsize if groupsize != -1 else infeatures
        self.maxq = 2 ** self.bits - 1
        G = math.ceil(infeatures / self.groupsize)
        self.register_buffer("qweight", torch.zeros((infeatures // 32 * bits, outfeatures), dtype=torch.int32))
        self.register_buffer("qzeros", torch.zeros((G, outfeatures // 32 * bits), dtype=torch.int32))
        self.register_buffer("scales", torch.zeros((G, outfeatures), dtype=torch.float16))
        self.register_buffer("g_idx", (torch.arange(infeatures, dtype=torch.int64) // self.groupsize).to(torch.int32))
        if bias:
            self.register_buffer("bias", torch.zeros((outfeatures,), dtype=torch.float16))
        else:
            self.bias = None
        # derived, non-persistent state built by post_init() on the device
        self._ready_for = None
        self._settled = None       # the _constants that a launch may read without waiting
        self._qweight_run = None   # the weights the kernels read: qweight itself or its row-sorted copy
        self._g_idx_run = None     # None => rows use group k // groupsize
        self._x_perm = None        # None => no gather of x
        self._gemv_rows = GEMV_MAX_M   # largest batch that goes through the GEMV
        self._gemm_ok = False      # the run-time layout meets the tensor-core kernel's one-group-per-32-rows rule
        # Row-parallel shard of a tensor-parallel model: forward_reduce() returns the sum over ranks.  `exchange` is an
        # exchange.PeerExchange (fused all-reduce for up to 8 rows), `tp_bias` the full bias that every rank adds after
        # the sum.
        self.exchange = None
        self.tp_bias = None
        # (slices_per_sm, ctas_per_sm) of b200gptq_gemv_tuned, or None for the library defaults
        self.gemv_tuning = None
        self._plans = {}           # (rows, tuning, activation) -> (ops.GemvPlan, the _constants it was made from)
        self._native = None        # _host.Layer: the prepared call in native code, made by the first forward

    # ---- offline packing (CPU) ----------------------------------------------------------
    def pack(self, linear, scales, zeros, g_idx=None):
        """Same contract as ``QuantLinear.pack`` of the reference (qlinear.py:77-175):
        ``scales`` / ``zeros`` are ``[outfeatures, G]``; the integer weight is
        ``round((W + zero*scale) / fp16(scale))`` per row group and ``zeros - 1`` is stored.
        With the layer and the statistics on a CUDA device the whole procedure runs there (the
        reference packs with a Python loop over the rows on the CPU); the result is bit-identical."""
        W = linear.weight.data
        if isinstance(linear, nn.Conv2d):
            W = W.flatten(1)
        elif type(linear).__name__ == "Conv1D":  # transformers.pytorch_utils.Conv1D keeps [in, out]
            W = W.t()
        rows = g_idx if g_idx is not None else self.g_idx
        # (contiguous tensors on one device: outputs, copy of g_idx and launch in one native call; 38 us of host work once, for 26 on the device)
        packed = _lib._host.pack(W, scales, zeros, rows, self.bits, g_idx is not None) if W.is_cuda else None
        if packed is not None:
            if linear.bias is not None:
                self.bias = linear.bias.detach().clone().half()
            self._store("qweight", packed[0])
            self._store("qzeros", packed[1])
            self._store("scales", packed[2])
            if g_idx is not None:
                self._store("g_idx", packed[3])
            self.__dict__["_ready_for"] = None
            return
        self.g_idx = g_idx.clone() if g_idx is not None else self.g_idx
        if ops.can_pack_linear(W, scales, zeros):
            if linear.bias is not None:
                self.bias = linear.bias.detach().clone().half()
            self.qweight, self.qzeros, self.scales = ops.pack_linear(W, scales.detach(), zeros.detach(), self.g_idx, self.bits)
            self._ready_for = None
            return
        g = self.g_idx.long()
        scales = scales.t().contiguous()
        zeros = zeros.t().contiguous()
        scale_zeros = zeros * scales
        self.scales = scales.clone().half()
        if linear.bias is not None:
            self.bias = linear.bias.detach().clone().half()
        intweight = torch.round((W.t() + scale_zeros[g]) / self.scales[g]).to(torch.int)
        if W.is_cuda:
            # statistics narrower than fp32: the same expression element by element, words built by b200gptq_pack_fields
            self.qweight = ops.pack_fields(intweight.contiguous(), self.bits)
            zq = (zeros - 1).to(torch.int64).to(torch.int32)
            self.qzeros = ops.pack_fields(zq.t().contiguous(), self.bits).t().contiguous()
            self._ready_for = None
            return
        intweight = torch.from_numpy(intweight.numpy().astype(np.uint32).astype(np.int64))
        self.qweight = _pack_fields(intweight, self.bits)
        zq = torch.from_numpy((zeros - 1).numpy().astype(np.uint32).astype(np.int64))
        self.qzeros = _pack_fields(zq.t().contiguous(), self.bits).t().contiguous()
        self._ready_for = None

    def _store(self, name: str, tensor) -> None:
        """``setattr`` of a buffer, without its 2 us where there is nothing else for it to do."""
        if name in self._buffers and name not in self._non_persistent_buffers_set and not _buffer_hooks:
            self._buffers[name] = tensor
        else:
            setattr(self, name, tensor)

    # ---- device-side preparation ----------------------------------------------------------
    def post_init(self):
        """Build the run-time view of the layer on its current device.

        A layer whose ``g_idx`` is constant over every aligned block of 32 rows is
        used as stored.  Any other ``g_idx`` (act-order checkpoints) is re-ordered
        once so that rows of a group are adjacent; ``forward`` then gathers ``x``
        through the permutation inside the kernels.
        """
        dev = self.qweight.device
        if dev.type != "cuda":
            raise RuntimeError("QuantLinear.post_init needs the module on a CUDA device")
        K = self.infeatures
        g = self.g_idx
        trivial = torch.equal(g, (torch.arange(K, device=dev, dtype=torch.int64) // self.groupsize).to(torch.int32))
        if trivial:
            self._qweight_run, self._g_idx_run, self._x_perm = self.qweight, None, None
        else:
            blocks = g.view(K // 32, 32)
            lo, hi = torch.aminmax(g)
            block_uniform, lo, hi = torch.stack([(blocks == blocks[:, :1]).all().to(g.dtype), lo, hi]).tolist()
            if lo < 0 or hi >= self.scales.shape[0]:
                raise ValueError(f"g_idx names group {lo if lo < 0 else hi}, the layer has {self.scales.shape[0]}")
            if block_uniform:
                self._qweight_run, self._g_idx_run, self._x_perm = self.qweight, g.contiguous(), None
            else:
                qs, perm, gs = ops.sort_rows(self.qweight.contiguous(), g.contiguous(), self.bits)
                sorted_trivial = torch.equal(
                    gs, (torch.arange(K, device=dev, dtype=torch.int64) // self.groupsize).to(torch.int32))
                self._qweight_run, self._x_perm = qs, perm
                self._g_idx_run = None if sorted_trivial else gs
        # true for every run-time g_idx built above (block-uniform, or sorted by group with whole blocks) except a sorted
        # layout whose groups do not fill whole blocks
        g_run, uniform = self._g_idx_run, True
        if g_run is not None:
            b = g_run.view(K // 32, 32)
            uniform = bool((b == b[:, :1]).all().item())
        self._gemm_ok, self._gemv_rows = row_rules(K, self.groupsize, g_run is not None, uniform)
        self._plans = {}
        self._native = None
        self._ready_for = self._stored()
        self._settled = self._constants()    # (the look at g_idx above has waited for the stream)

    def _stored(self):
        """What the run-time view was built from: where the stored weights and groups lie, on whatever device, and how often
        they have been written to (weights that the kernels read as stored may be)."""
        q, g = self._buffers["qweight"], self._buffers["g_idx"]
        return q.data_ptr(), g.data_ptr(), 0 if self._qweight_run is q else _version(q), _version(g)

    def _ready(self) -> bool:
        return self._ready_for == self._stored()

    def __getstate__(self):
        """For ``copy.deepcopy`` and ``torch.save``: prepared launches hold addresses of this process and are made anew."""
        state = dict(self.__dict__, _plans={}, _native=None, _ready_for=None, _settled=None)
        for name in ("_native_state", "_native_tuning"):
            state.pop(name, None)
        return state

    # ---- forward --------------------------------------------------------------------------
    def forward(self, x):
        if torch.compiler.is_compiling():
            # Traced: one opaque, shape-inferable operator per layer (torch_ops.py).  The run-time layout must exist
            # already (post_init(), which from_quantized and the first eager call run); the prepared plans below are
            # for eager calls.
            from .torch_ops import quant_matmul
            x2 = x.half().reshape(-1, self.infeatures).contiguous()
            y = quant_matmul(x2, self._qweight_run, self.qzeros, self.scales, self._g_idx_run, self._x_perm,
                             self.bias, self.bits, self.groupsize, self._gemm_ok)
            return y.reshape(x.shape[:-1] + (self.outfeatures,))
        native = self._native
        if native is not None:
            # fp16, contiguous, on the layer's device, prepared before: checks, allocation and launch in one native call
            y = native.run(x, self.__dict__)
            if y is not None:
                return y
        if not x.is_cuda:
            raise RuntimeError("QuantLinear.forward needs CUDA tensors: this backend has no CPU path")
        if not self._ready():
            self.post_init()
        out_shape = x.shape[:-1] + (self.outfeatures,)
        x2 = x.half().reshape(-1, x.shape[-1])
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        M = x2.shape[0]
        now = self._constants()
        self._settle(now)
        qzeros, scales, bias = now[:3]
        kw = dict(bias=bias, x_perm=self._x_perm)
        args = (self._qweight_run, qzeros, scales, self._g_idx_run, self.bits, self.groupsize)
        if M <= self._gemv_rows:
            plan = self._plan(M, now)
            y = self._prepare_native(now, x2, M, plan)
            if y is None:
                with torch.cuda.device(x2.device):
                    y = plan.run(x2)
        elif self._gemm_ok:
            # above that one tensor-core pass beats several GEMV passes
            y = self._prepare_native(now, x2)
            if y is None:
                y = ops.gemm(x2, *args, **kw)
        elif M > 64:
            # no tensor-core kernel for this layout and many rows: dequantise once with the library's kernel (the
            # reference's own dequantise-then-matmul order, qlinear.py:242-243) and let the dense product run on the
            # GPU's GEMM library; M / 8 GEMV passes would read the weights M / 8 times
            _, W = ops.dequantize(self._qweight_run, self.qzeros, self.scales, self._g_idx_run, self.bits,
                                  self.groupsize, want_q=False)
            xg = x2 if self._x_perm is None else x2.index_select(1, self._x_perm.long())
            y = xg @ W
            if self.bias is not None:
                y = y + self.bias
        else:
            # layers whose groups cut through 32-row blocks have no tensor-core kernel: GEMV passes of up to 8 rows
            y = torch.empty((M, self.outfeatures), dtype=torch.float16, device=x2.device)
            for m0 in range(0, M, GEMV_MAX_M):
                ops.gemv(x2[m0:m0 + GEMV_MAX_M], *args, out=y[m0:m0 + GEMV_MAX_M], **kw)
        return y.reshape(out_shape)

    def _constants(self):
        """What a prepared launch holds beside the rows themselves: these tensors, where their numbers lie (``.data`` may
        have been replaced) and how often they have been written to."""
        b = self._buffers
        qzeros, scales, bias = b["qzeros"], b["scales"], b.get("bias", self.__dict__.get("bias"))
        return (qzeros, scales, bias, qzeros.data_ptr(), scales.data_ptr(), None if bias is None else bias.data_ptr(),
                _version(qzeros), _version(scales), _version(b["qweight"]))

    def _settle(self, now):
        """The kernels read weights, scales and zero-points before the kernel in front of them has ended.  Where those are new since
        the last call, what wrote them may be that kernel: something that waits for it comes in between."""
        if self._settled is None or not _same(self._settled, now):
            ops.settle(self._buffers["qweight"].device)
            self._settled = now

    def _plan(self, rows: int, now, input_act: int = 0):
        """The prepared GEMV of this row count, made anew when a tensor that it points to is not the one in ``now``
        (``_constants``) any more."""
        key = (rows, self.gemv_tuning, input_act)
        made = self._plans.get(key)
        if made is None or not _same(made[1], now):
            plan = ops.GemvPlan(self._qweight_run, now[0], now[1], self._g_idx_run, self._x_perm, now[2], rows, self.bits,
                                self.groupsize, self.gemv_tuning, input_act)
            made = self._plans[key] = (plan, now)
        return made[0]

    def _prepare_native(self, now, x2, rows: int = 0, plan=None):
        """Make the native call object for the current buffers (once), hand it the plan of one more row count, and make the
        call; None where it does not take it (a tensor that is not a plain one, another current device)."""
        device = self._buffers["qweight"].device
        if device.type != "cuda":
            return None
        if self._native is None or not _same(self._native_state, now) or self._native_tuning is not self.gemv_tuning:
            self._native_state, self._native_tuning = now, self.gemv_tuning
            self._native = _lib._host.Layer(self.infeatures, self.outfeatures, self.bits, self.groupsize,
                                            device.index, self.__dict__, self._gemm_ok, self._gemv_rows,
                                            self._qweight_run, self._g_idx_run, self._x_perm)
        if plan is not None:
            self._native.set_gemv(rows, plan, plan._handle.value, plan._need)
        return self._native.run(x2, self.__dict__)

    # ---- the element-wise kernel in front of this layer folded into its read of x (decode batches only) ----
    def can_fold(self, rows: int, input_act: int) -> bool:
        """Whether :meth:`forward_act` / ``forward_reduce(..., input_act)`` can take the activation for ``rows`` rows."""
        if not self._ready():
            self.post_init()
        return rows <= GEMV_MAX_M and ops.can_fold_act(rows, self.infeatures, self.outfeatures, self.bits, self.groupsize,
                                                       self._g_idx_run is not None, self._x_perm is not None, input_act)

    def forward_act(self, u, input_act: int):
        """``forward(act(u))`` in one launch for up to 8 rows: ``input_act = _lib.ACT_SWIGLU`` (``u`` is
        ``[..., 2 * in] = [gate | up]``) or ``_lib.ACT_RELU`` (``b200gptq_gemv_plan_create_ex``).  The caller checks
        :meth:`can_fold` first."""
        if not self._ready():
            self.post_init()
        u2 = u.half().reshape(-1, u.shape[-1])
        if not u2.is_contiguous():
            u2 = u2.contiguous()
        M = u2.shape[0]
        now = self._constants()
        self._settle(now)
        plan = self._plan(M, now, input_act)
        with torch.cuda.device(u2.device):
            y = plan.run(u2)
        return y.reshape(u.shape[:-1] + (self.outfeatures,))

    def forward_reduce(self, x, input_act: int = 0):
        """Row-parallel forward: this rank's slice of the input in, the complete output (summed over ranks) out.
        Up to 8 rows go through ``b200gptq_gemv_tp`` (sum fused into the kernel, peer memory); more rows use the
        process group's all-reduce."""
        if self.exchange is None:
            raise RuntimeError("forward_reduce needs an exchange (see exchange.PeerExchange)")
        if not self._ready():
            self.post_init()
        x2 = x.half().reshape(-1, x.shape[-1])
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        if x2.shape[0] <= GEMV_MAX_M:
            self._settle(self._constants())
            y = ops.gemv_tp(x2, self._qweight_run, self.qzeros, self.scales, self._g_idx_run, self.bits, self.groupsize,
                            self.exchange, bias=self.tp_bias, x_perm=self._x_perm, tuning=self.gemv_tuning,
                            input_act=input_act)
        else:
            if input_act:
                raise ValueError("an input activation is folded for up to 8 rows only")
            import torch.distributed as dist
            saved, self.bias = self.bias, None
            try:
                y = self.forward(x2)
            finally:
                self.bias = saved
            dist.all_reduce(y, group=self.exchange.group)
            if self.tp_bias is not None:
                y = y + self.tp_bias
        return y.reshape(x.shape[:-1] + (self.outfeatures,))

    def extra_repr(self):
        return (f"in={self.infeatures}, out={self.outfeatures}, bits={self.bits}, "
                f"groupsize={self.groupsize}, bias={self.bias is not None}")


__all__ = ["QuantLinear"]
