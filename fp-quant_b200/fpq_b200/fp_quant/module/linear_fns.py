"""Forward functions of the quantised linear layer, mirroring
inference_lib/src/fp_quant/module/linear_fns.py (IST-DASLab/FP-Quant): `forward_quantize`,
`forward_gemm`, the two bf16-backward autograd functions and the MXFP8-backward pair
(`FPQuant4x8MasterFn`: both gradient GEMMs on MXFP8 operands).  Backward through pre-quantised
weights raises like the reference does.  `FPQuant4x4MasterFn` runs both gradient GEMMs on MXFP4 operands.
"""
from __future__ import annotations

from typing import Callable, Optional, Tuple

import torch
from torch.autograd import Function

from ..utils.config import FPQuantDtype
from ... import ops
from ...ops import plain_eager
from ...rotation import kind_of
from .qutlass_ops import (backward_bf16_square_double_mxfp8_op, backward_qt_bf16_op, backward_t_bf16_op,
                          fused_quantize_blocked_op, fused_quantize_mx_op,
                          fused_quantize_nv_op, matmul_fp4_bf16_tn_blocked_op, matmul_mxf4_bf16_tn_op,
                          matmul_mxf8_bf16_nn_op, matmul_mxf8_bf16_tn_op, matmul_nvf4_bf16_tn_op,
                          mxfp4_transpose_mxfp8_op)


class GemmConstants:
    """fp32 [1] tensors that follow from the two tensor scales: `alpha` (`gemm_alpha`), the scales themselves, and for the
    MXFP8 backward their inverses, made when they are first asked for."""

    @torch.no_grad()
    def __init__(self, weight_global_scale: torch.Tensor, act_global_scale: torch.Tensor, own: bool = False):
        """`own`: never the storage of fp32 scales themselves, so that `update` can be called."""
        self.alpha = gemm_alpha(weight_global_scale, act_global_scale)
        self.weight_scale, self.act_scale = (s.to(torch.float32, copy=own).reshape(1)
                                             for s in (weight_global_scale, act_global_scale))
        self._inverses = None

    @torch.no_grad()
    def update(self, weight_global_scale: torch.Tensor, act_global_scale: torch.Tensor) -> None:
        """The same tensors with the values of other scales."""
        self.alpha.copy_(gemm_alpha(weight_global_scale, act_global_scale))
        self.weight_scale.copy_(weight_global_scale.reshape(1))
        self.act_scale.copy_(act_global_scale.reshape(1))
        self._inverses = None

    @torch.no_grad()
    def inverses(self) -> Tuple[torch.Tensor, torch.Tensor]:
        """(1 / act_scale, 1 / weight_scale).  Not kept when the stream is being captured: a graph's tensors hold nothing
        before it is replayed."""
        if self._inverses is not None:
            return self._inverses
        pair = (1.0 / self.act_scale, 1.0 / self.weight_scale)
        if not torch.cuda.is_current_stream_capturing():
            self._inverses = pair
        return pair


class ConstantsCache:
    """`GemmConstants` of one layer, remade only when one of its two tensor scales changed (up to nine small kernels per
    training step otherwise).  The tensors a set was made from are kept and compared as objects, so an address that is used
    again cannot pass for them.  One set per stream, so that no stream reads what another one may not have written yet.
    Nothing made while the stream is being captured is kept: its values only exist after a replay."""
    STREAMS = 64        # torch hands out 32 streams a priority in turn; a set is three blocks of 512 bytes

    def __init__(self):
        self._training = None       # (scales, {stream: set}), replaced as a whole: threads see one state or the other
        self._inference = {}        # stream: [scales, set], the sets for as long as the layer lives

    @staticmethod
    def _same(of, w: torch.Tensor, a: torch.Tensor) -> bool:
        return (of[0] is w and of[1] is a and of[2] == w._version and of[3] == a._version and of[4] == w.data_ptr()
                and of[5] == a.data_ptr())

    @staticmethod
    def _of(w: torch.Tensor, a: torch.Tensor):
        return (w, a, w._version, a._version, w.data_ptr(), a.data_ptr())

    def training(self, w: torch.Tensor, a: torch.Tensor, stream: int, capturing: bool) -> GemmConstants:
        """A set that stays as it is, since a backward pass may hold it.  A captured step derives its own inside the graph:
        replays follow updates of the scales in place, and no graph holds an address in here."""
        if capturing:
            return GemmConstants(w, a)
        state = self._training
        if state is None or not self._same(state[0], w, a):
            state = self._training = (self._of(w, a), {})
        kept = state[1]
        consts = kept.get(stream)
        if consts is None:
            if len(kept) >= self.STREAMS:
                kept.clear()
            consts = kept[stream] = GemmConstants(w, a)
        return consts

    def inference(self, w: torch.Tensor, a: torch.Tensor, stream: int, capturing: Callable[[], bool]) -> GemmConstants:
        """A set that CUDA graphs may hold the addresses of: captured passes take an earlier pass's, which costs their replays
        nothing.  It is therefore never dropped, and new scales are written into it.  `capturing` is only asked where this
        stream's set does not fit (the question costs a decode step a microsecond)."""
        entry = self._inference.get(stream)
        if entry is not None and self._same(entry[0], w, a):
            return entry[1]
        if capturing():
            for of, consts in list(self._inference.values()):
                if self._same(of, w, a):
                    return consts
            return GemmConstants(w, a)
        if entry is not None and entry[1].alpha.device == w.device:
            entry[1].update(w, a)
            entry[0] = self._of(w, a)
            return entry[1]
        consts = GemmConstants(w, a, own=True)
        if entry is not None or len(self._inference) < self.STREAMS:
            self._inference[stream] = [self._of(w, a), consts]
        return consts


def forward_quantize(x: torch.Tensor, hadamard_matrix: torch.Tensor, global_scale: torch.Tensor,
                     dtype: FPQuantDtype, forward_method: str) -> Tuple[torch.Tensor, torch.Tensor, Optional[torch.Tensor]]:
    """rotate + quantise -> (codes, row-major padded scales, mask) (linear_fns.py:27-50)."""
    if dtype == FPQuantDtype.MXFP4:
        return fused_quantize_mx_op(x.to(torch.bfloat16), hadamard_matrix.to(torch.bfloat16), forward_method,
                                    forward_method == "quest" and x.requires_grad)
    if dtype == FPQuantDtype.NVFP4:
        q, s = fused_quantize_nv_op(x.to(torch.bfloat16), hadamard_matrix.to(torch.bfloat16), global_scale.float())
        return q, s, None
    raise ValueError(f"Unsupported forward dtype: {dtype}")


def forward_gemm(x_q, w_q, x_scales, w_scales, alpha, dtype: FPQuantDtype):
    """bf16 = alpha * dq(x_q) dq(w_q)^T from row-major scales (linear_fns.py:53-64)."""
    if dtype == FPQuantDtype.MXFP4:
        return matmul_mxf4_bf16_tn_op(x_q, w_q, x_scales, w_scales, alpha.float())
    if dtype == FPQuantDtype.NVFP4:
        return matmul_nvf4_bf16_tn_op(x_q, w_q, x_scales, w_scales, alpha.float())
    raise ValueError(f"Unsupported dtype: {dtype}")


def forward_quantize_blocked(x, hadamard_matrix, global_scale, dtype: FPQuantDtype, forward_method: str,
                             rotation: int = 0):
    """Fast path of `forward_quantize`: scales come out in the layout the matmul reads."""
    if dtype not in (FPQuantDtype.MXFP4, FPQuantDtype.NVFP4):
        raise ValueError(f"Unsupported forward dtype: {dtype}")
    if forward_method not in ("abs_max", "quest"):
        raise ValueError(f"Unsupported forward method: {forward_method}")
    return fused_quantize_blocked_op(x.to(torch.bfloat16), hadamard_matrix.to(torch.bfloat16), global_scale.float(),
                                     dtype == FPQuantDtype.NVFP4, rotation, forward_method == "quest")


def forward_gemm_blocked(x_q, w_q, x_scales_blocked, w_scales_blocked, alpha, dtype: FPQuantDtype, bias=None):
    if dtype not in (FPQuantDtype.MXFP4, FPQuantDtype.NVFP4):
        raise ValueError(f"Unsupported dtype: {dtype}")
    return matmul_fp4_bf16_tn_blocked_op(x_q, w_q, x_scales_blocked, w_scales_blocked, alpha.float(),
                                         dtype == FPQuantDtype.NVFP4, bias)


def gemm_alpha(weight_global_scale: torch.Tensor, act_global_scale: torch.Tensor) -> torch.Tensor:
    """fp32 [1]: 1 / (weight_global_scale * act_global_scale) with the reference's rounding order -- product
    and reciprocal in the dtype of the buffers (bf16 once `pre_forward` made them), then the cast to fp32
    (linear_fns.py:433, :505 and `alpha.float()` at :57-62).  For the abs_max default 3 * 3 this is
    bf16(1/9) = 0.111328, not 0.111111."""
    return (1.0 / (weight_global_scale * act_global_scale)).float().reshape(1)


def _linear_forward(x, weight_q, weight_scales_blocked, weight_global_scale, act_global_scale, bias,
                    hadamard_matrix, dtype, forward_method, alpha=None):
    x_flat = x.contiguous().flatten(end_dim=-2)
    x_q, x_scales = forward_quantize_blocked(x_flat, hadamard_matrix, act_global_scale, dtype, forward_method)
    if alpha is None:
        alpha = gemm_alpha(weight_global_scale, act_global_scale)
    # the bias is added in the GEMM's epilogue (fp32 accumulator + bias, one rounding to bf16) instead of
    # the reference's separate bf16 add (linear_fns.py:514-515)
    fused_bias = bias if bias is not None and bias.dtype == torch.bfloat16 else None
    y = forward_gemm_blocked(x_q, weight_q, x_scales, weight_scales_blocked, alpha, dtype, fused_bias)
    y = y.unflatten(dim=0, sizes=x.shape[:-1])
    if bias is not None and fused_bias is None:
        y = y + bias
    return y


class FPQuant4x16NoMasterFn(Function):
    """Inference forward with pre-quantised weights (linear_fns.py:482-528).  `weight_scales` are
    the weight scale bytes already in the swizzled layout (cached by the module)."""

    @staticmethod
    def forward(ctx, x, weight_q, weight_scales, weight_global_scale, act_global_scale, bias,
                forward_hadamard_matrix, dtype, forward_method, alpha=None):
        """`alpha` (optional, fp32 [1]): the module's cached `gemm_alpha` of the two tensor scales."""
        return _linear_forward(x, weight_q, weight_scales, weight_global_scale, act_global_scale, bias,
                               forward_hadamard_matrix, dtype, forward_method, alpha)

    @staticmethod
    def backward(ctx, grad_output):
        raise NotImplementedError("Backward pass is not implemented for FPQuant4x16NoMasterFn yet")


class FPQuant4x16MasterFn(Function):
    """Forward quantises the bf16 master weight on the fly; backward is plain bf16
    (linear_fns.py:405-479)."""

    @staticmethod
    def forward(ctx, x, weight, weight_global_scale, act_global_scale, bias, forward_hadamard_matrix, dtype,
                forward_method, constants: Optional[GemmConstants] = None):
        """`constants` (optional): what follows from the two tensor scales, made once by the module."""
        alpha = None
        if constants is not None:
            alpha, act_global_scale, weight_global_scale = constants.alpha, constants.act_scale, constants.weight_scale
        w_q, w_scales = forward_quantize_blocked(weight, forward_hadamard_matrix, weight_global_scale, dtype,
                                                 forward_method)
        y = _linear_forward(x, w_q, w_scales, weight_global_scale, act_global_scale, bias,
                            forward_hadamard_matrix, dtype, forward_method, alpha)
        ctx.x_shape, ctx.bias_present = x.shape, bias is not None
        ctx.save_for_backward(x.contiguous().flatten(end_dim=-2), weight)
        return y

    @staticmethod
    def backward(ctx, grad_output):
        x_flat, weight = ctx.saved_tensors
        g = grad_output.flatten(end_dim=-2)
        grad_input = (g @ weight).view(ctx.x_shape)
        grad_weight = g.t() @ x_flat
        grad_bias = g.sum(dim=0) if ctx.bias_present else None
        return grad_input, grad_weight, None, None, grad_bias, None, None, None, None


def _unpack_mask(clip_mask: torch.Tensor) -> torch.Tensor:
    """[.., K/8] bytes -> [.., K] bool, bit i of byte b = element 8 b + i (linear_fns.py:67-77)."""
    bits = (clip_mask.unsqueeze(-1) >> torch.arange(8, device=clip_mask.device, dtype=torch.uint8)) & 1
    return bits.flatten(start_dim=-2).bool()


def _unrotate(g: torch.Tensor, mask: Optional[torch.Tensor], hadamard_matrix: torch.Tensor) -> torch.Tensor:
    """`(g * _unpack_mask(mask)).view(-1, h) @ hadamard_matrix.T` in bf16 (linear_fns.py:321-324): gradient with
    respect to the rotated operand -> gradient with respect to the operand, clipped elements without one.  The
    normalised Sylvester matrix is symmetric, so the butterfly kernel does it, with the mask applied to its input;
    any other matrix takes the dense product."""
    kind, group = kind_of(0, hadamard_matrix)
    if kind == "dense":
        if mask is not None:
            g = g * _unpack_mask(mask).view_as(g).to(g.dtype)
        return ops.rotate_dense(g.contiguous(), hadamard_matrix.t().contiguous(), out_dtype=torch.bfloat16)
    if mask is not None:
        return ops.rotate_hadamard_masked(g, mask, group if kind == "hadamard" else 0)
    return g if kind == "identity" else ops.rotate_hadamard(g.contiguous(), group, out_dtype=torch.bfloat16)


def _row_major_scales(scales: torch.Tensor, rows: int, sf_cols: int) -> torch.Tensor:
    sb = scales.view(torch.uint8)
    return sb if tuple(sb.shape) == (rows, sf_cols) else sb[:rows, :sf_cols].contiguous()


def _mxfp8_backward(grad_output, x_q, w_q, x_scales, w_scales, act_global_scale, weight_global_scale, x_mask, w_mask,
                    hadamard_matrix, x_shape, want_weight_grad: bool, swizzled: bool = False, constants=None):
    """The two gradient GEMMs of linear_fns.py:270-350 on MXFP8 operands.  The saved MXFP4 operands are
    transposed into MXFP8 (exactly, unless the scales of a 32-row band differ by more than 2^14), the bf16
    gradient is quantised once with a scale per 32 x 32 square and read along either axis.

    Same data flow as the reference's `mxfp4_transpose_mxfp8_op` / `backward_bf16_square_double_mxfp8_op` /
    `matmul_mxf8_bf16_tn_op` / `..._nn_op` sequence, with the re-layouts folded into the producers: the
    quantisers write their scales in the layout the GEMM reads, and the gradient's bytes come out in both
    orientations, so the `nn` product is a `tn` product of the transposed copy.  `swizzled`: x_scales and w_scales
    already are in the layout the GEMM reads."""
    if constants is not None:
        act_inverse, weight_inverse = constants.inverses()
    else:
        act_inverse, weight_inverse = ((1.0 / s.float()).reshape(1) for s in (act_global_scale, weight_global_scale))

    def operand_scales(scales, rows):
        return scales.view(torch.uint8) if swizzled else _row_major_scales(scales, rows, in_features // 32)

    g = grad_output.flatten(end_dim=-2).to(torch.bfloat16).contiguous()
    tokens, out_features = g.shape
    in_features = w_q.size(-1) * 2
    g_fp8, g_row_scales, g_col_scales, g_t_fp8 = ops.quantize_mxfp8_square(g, swizzled=True, transposed=want_weight_grad) \
        if want_weight_grad else ops.quantize_mxfp8_square(g, swizzled=True) + (None,)
    if out_features % 128 == 0:
        w_t_fp8, w_t_scales = ops.mxfp4_transpose_mxfp8(w_q.view(torch.uint8), operand_scales(w_scales, out_features), swizzled=True,
                                                        scales_swizzled=swizzled)
    else:     # the transposed weight is padded along the contraction axis: cut it back to the gradient's width
        w_t_fp8, w_t_scales = ops.mxfp4_transpose_mxfp8(w_q.view(torch.uint8), operand_scales(w_scales, out_features), scales_swizzled=swizzled)
        w_t_fp8 = w_t_fp8[:, :out_features].contiguous()
        w_t_scales = ops.swizzle_scales(w_t_scales[:, : out_features // 32].contiguous())
    grad_input = ops.gemm_mxf8(g_fp8, w_t_fp8, g_row_scales, w_t_scales, weight_inverse)[:tokens]
    grad_input = _unrotate(grad_input, x_mask, hadamard_matrix).view(x_shape)
    grad_weight = None
    if want_weight_grad:
        x_t_fp8, x_t_scales = ops.mxfp4_transpose_mxfp8(x_q.view(torch.uint8), operand_scales(x_scales, tokens), swizzled=True,
                                                        scales_swizzled=swizzled)                       # [in, tokens_up128]
        grad_weight = ops.gemm_mxf8(g_t_fp8, x_t_fp8, g_col_scales, x_t_scales, act_inverse)
        grad_weight = _unrotate(grad_weight, w_mask, hadamard_matrix).view(out_features, in_features)
    return grad_input, grad_weight


def _training_forward(x, weight, weight_global_scale, act_global_scale, bias, hadamard_matrix, dtype, forward_method,
                      constants: Optional[GemmConstants], mxfp4_backward: bool = False):
    """Forward pass of the MXFP4 layers whose backward runs on quantised operands: (y, (codes, scales, clip mask) of x and
    of the weight, whether the scales are swizzled).  Where the calls need not be traced and the backward (the MXFP4 one has
    a general form) reads the scales so, the kernels are called directly and the scales stay in the layout that the
    matmul reads; otherwise the reference's op sequence with its row-major scales.  The rotation is classified once: that
    waits for the GPU where the matrix has to be converted (weights that are not bf16)."""
    x_flat = x.contiguous().flatten(end_dim=-2)
    matrix = hadamard_matrix.to(torch.bfloat16)
    direct = (constants is not None and dtype == FPQuantDtype.MXFP4 and forward_method in ("abs_max", "quest")
              and plain_eager(x) and plain_eager(weight))
    if direct:
        kind, group = kind_of(0, matrix)
        direct = kind != "dense" and (not mxfp4_backward or _fused_mxfp4_backward(kind, group, weight.shape[0]))
    if direct:
        group = group if kind == "hadamard" else 0

        def quantize(t):
            t16 = t.to(torch.bfloat16)
            if forward_method == "quest":
                return ops.quantize_quest(t16, group, swizzled=True, return_mask=t.requires_grad)
            return ops.quantize(t16, "mxfp4", group, None, swizzled=True)[:2] + (None,)

        xq, wq = quantize(x_flat), quantize(weight)
        y = ops.gemm_fp4(xq[0], wq[0], xq[1], wq[1], constants.alpha, "mxfp4")
    else:
        xq = forward_quantize(x_flat, matrix, act_global_scale, dtype, forward_method)
        wq = forward_quantize(weight, matrix, weight_global_scale, dtype, forward_method)
        y = forward_gemm(xq[0], wq[0], xq[1], wq[1], 1.0 / (weight_global_scale * act_global_scale), dtype)
    y = y.unflatten(dim=0, sizes=x.shape[:-1])
    if bias is not None:
        y = y + bias
    return y, xq, wq, direct


def _fused_mxfp4_backward(kind: str, group: int, out_features: int) -> bool:
    """Whether the MXFP4 backward runs on the transposing kernels: a rotation that fits a scale group, rows they can load."""
    return kind in ("hadamard", "identity") and group <= 32 and out_features % 8 == 0


class FPQuant4x8MasterFn(Function):
    """MXFP4 forward from a bf16 master weight, MXFP8 backward (linear_fns.py:232-350)."""

    @staticmethod
    def forward(ctx, x, weight, weight_global_scale, act_global_scale, bias, forward_hadamard_matrix, dtype,
                forward_method, constants: Optional[GemmConstants] = None):
        y, (x_q, x_scales, x_mask), (w_q, w_scales, w_mask), ctx.swizzled = _training_forward(
            x, weight, weight_global_scale, act_global_scale, bias, forward_hadamard_matrix, dtype, forward_method, constants)
        ctx.x_shape, ctx.bias_present, ctx.constants = x.shape, bias is not None, constants
        ctx.masks = (x_mask, w_mask)
        ctx.save_for_backward(x_q, w_q, x_scales, w_scales, act_global_scale, weight_global_scale, forward_hadamard_matrix)
        return y

    @staticmethod
    def backward(ctx, grad_output):
        x_q, w_q, x_scales, w_scales, act_global_scale, weight_global_scale, hadamard_matrix = ctx.saved_tensors
        x_mask, w_mask = ctx.masks
        grad_input, grad_weight = _mxfp8_backward(grad_output, x_q, w_q, x_scales, w_scales, act_global_scale,
                                                  weight_global_scale, x_mask, w_mask, hadamard_matrix, ctx.x_shape, True,
                                                  ctx.swizzled, ctx.constants)
        grad_bias = grad_output.flatten(end_dim=-2).sum(dim=0) if ctx.bias_present else None
        return grad_input, grad_weight, None, None, grad_bias, None, None, None, None


class FPQuant4x8NoMasterFn(Function):
    """MXFP4 forward from pre-quantised weights (row-major scale bytes as stored in a checkpoint); the
    backward raises, as the reference's does (linear_fns.py:352-404)."""

    @staticmethod
    def forward(ctx, x, weight_q, weight_scales, weight_global_scale, act_global_scale, bias, forward_hadamard_matrix,
                dtype, forward_method):
        x_flat = x.contiguous().flatten(end_dim=-2)
        x_q, x_scales, _ = forward_quantize(x_flat, forward_hadamard_matrix, act_global_scale, dtype, forward_method)
        y = forward_gemm(x_q, weight_q, x_scales, weight_scales, 1.0 / (weight_global_scale * act_global_scale), dtype)
        y = y.unflatten(dim=0, sizes=x.shape[:-1])
        if bias is not None:
            y = y + bias
        return y

    @staticmethod
    def backward(ctx, grad_output):
        raise NotImplementedError("Backward pass is not implemented for FPQuant4x8NoMasterFn yet")


class FPQuant4x4MasterFn(Function):
    """MXFP4 forward from a bf16 master weight, MXFP4 backward (linear_fns.py:80-230): the gradient and the
    dequantised, transposed operands are rotated along the contraction axis with the Hadamard matrix,
    quantised to MXFP4 again (abs_max), and both gradient GEMMs run on the FP4 kernel."""

    @staticmethod
    def forward(ctx, x, weight, weight_global_scale, act_global_scale, bias, forward_hadamard_matrix, dtype,
                forward_method, constants: Optional[GemmConstants] = None):
        y, (x_q, x_scales, x_mask), (w_q, w_scales, w_mask), ctx.swizzled = _training_forward(
            x, weight, weight_global_scale, act_global_scale, bias, forward_hadamard_matrix, dtype, forward_method, constants,
            mxfp4_backward=True)
        ctx.x_shape, ctx.bias_present, ctx.constants = x.shape, bias is not None, constants
        ctx.masks = (x_mask, w_mask)
        ctx.save_for_backward(x_q, w_q, x_scales, w_scales, act_global_scale, weight_global_scale, forward_hadamard_matrix)
        return y

    @staticmethod
    def backward(ctx, grad_output):
        x_q, w_q, x_scales, w_scales, act_global_scale, weight_global_scale, hadamard_matrix = ctx.saved_tensors
        x_mask, w_mask = ctx.masks
        # The reference multiplies the columns of the Hadamard matrix by fresh random signs here
        # (linear_fns.py:151-158).  With y = x @ (H D) that flips the sign of whole columns of both rotated
        # operands of a GEMM, which neither the sign-symmetric quantiser nor the product of the two notices:
        # both gradients are bit-identical with D = I.  The plain matrix is used, so the rotation stays on the
        # butterfly of the quantise kernel instead of a dense product.
        backward_hadamard_matrix = hadamard_matrix.to(torch.bfloat16)
        g = grad_output.flatten(end_dim=-2).to(torch.bfloat16).contiguous()
        tokens, out_features = g.shape
        in_features = w_q.size(-1) * 2
        # abs_max MXFP4 carries a factor 3 per operand (the scale is a third of the power of two that is stored)
        ninth = torch.full((1,), 1.0 / 9.0, dtype=torch.float32, device=g.device)
        kind, group = kind_of(0, backward_hadamard_matrix)
        if _fused_mxfp4_backward(kind, group, out_features):
            # Same data flow as the op sequence below with the re-layouts folded into the producers: scales come
            # out in the layout the GEMM reads, the transposes happen inside the (de)quantise kernels, and the
            # token axis is padded to a whole number of K tiles by the kernels that write it.
            gh = group if kind == "hadamard" else 0
            swz, consts = ctx.swizzled, ctx.constants
            w_sc, x_sc = (w_scales, x_scales) if swz else (_row_major_scales(w_scales, out_features, in_features // 32),
                                                           _row_major_scales(x_scales, tokens, in_features // 32))
            w_gs, x_gs = (consts.weight_scale, consts.act_scale) if consts is not None else (weight_global_scale.float(),
                                                                                              act_global_scale.float())
            g_q, g_s, _ = ops.quantize(g, "mxfp4", gh, None, swizzled=True)
            wt_q, wt_s = ops.mxfp4_requantize_transposed(w_q.view(torch.uint8), w_sc, w_gs, gh, swizzled=True,
                                                         scales_swizzled=swz)                                     # [in, out]
            grad_input = ops.gemm_fp4(g_q, wt_q, g_s, wt_s, ninth, "mxfp4")
            gt_q, gt_s = ops.quantize_transposed(g, gh, pad_to=128, swizzled=True)                             # [out, tokens_up128]
            xt_q, xt_s = ops.mxfp4_requantize_transposed(x_q.view(torch.uint8), x_sc, x_gs, gh, pad_to=128, swizzled=True,
                                                         scales_swizzled=swz)                                     # [in, tokens_up128]
            grad_weight = ops.gemm_fp4(gt_q, xt_q, gt_s, xt_s, ninth, "mxfp4")
        else:
            g_q, g_scales, _ = fused_quantize_mx_op(g, backward_hadamard_matrix, "abs_max", False)
            wt_q, wt_scales = backward_qt_bf16_op(w_q, w_scales, backward_hadamard_matrix, weight_global_scale.float())
            grad_input = matmul_mxf4_bf16_tn_op(g_q, wt_q, g_scales, wt_scales, ninth)
            # the weight gradient contracts over the tokens: pad them to a whole number of K tiles with zero rows
            pad = (-tokens) % 128
            g_pad = torch.nn.functional.pad(g, (0, 0, 0, pad)) if pad else g
            gt_q, gt_scales = backward_t_bf16_op(g_pad, backward_hadamard_matrix)
            if pad:
                zero_codes = torch.full((pad, x_q.shape[1]), 0x88, dtype=torch.uint8, device=x_q.device)
                x_q_pad = torch.cat([x_q.view(torch.uint8), zero_codes])
                xs = x_scales.view(torch.uint8)[:tokens, : x_q.shape[1] // 16]
                xs_pad = torch.cat([xs, torch.full((pad, xs.shape[1]), 127, dtype=torch.uint8, device=xs.device)])
            else:
                x_q_pad, xs_pad = x_q, x_scales
            xt_q, xt_scales = backward_qt_bf16_op(x_q_pad, xs_pad, backward_hadamard_matrix, act_global_scale.float())
            grad_weight = matmul_mxf4_bf16_tn_op(gt_q, xt_q, gt_scales, xt_scales, ninth)
        grad_input = _unrotate(grad_input, x_mask, hadamard_matrix).view(ctx.x_shape)
        grad_weight = _unrotate(grad_weight, w_mask, hadamard_matrix).view(out_features, in_features)
        grad_bias = g.sum(dim=0) if ctx.bias_present else None
        return grad_input, grad_weight, None, None, grad_bias, None, None, None, None
