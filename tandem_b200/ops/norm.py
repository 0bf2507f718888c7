"""LayerNorm on the fused kernels (tandem_b200/cuda/layers.cu): one pass forward
saving mean and 1/std per row; one pass backward producing dx plus per-block
partial sums of the weight and bias gradients, reduced in a fixed order."""

import torch

from ._lib import check_rc, direct, lib, need, need_bf16, run, stream, vectors_of


class _LayerNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, b, eps):
        need_bf16(x, w, b)
        need(x.dim() > 0 and w.numel() == x.shape[-1] == b.numel(), "layer_norm takes a weight and a bias with one value per column")
        x2 = vectors_of(x.reshape(-1, x.shape[-1]))
        gain, shift = vectors_of(w), vectors_of(b)
        M, D = x2.shape
        y = torch.empty_like(x2)
        stats = torch.empty(2, M, dtype=torch.float32, device=x.device)  # the rows' mean and 1 / std
        check_rc(lib().tb_layernorm_fwd(x2.data_ptr(), gain.data_ptr(), shift.data_ptr(), y.data_ptr(), stats.data_ptr(), stats.data_ptr() + 4 * M,
                                        M, D, eps, stream(x)), "layernorm forward")
        ctx.save_for_backward(x2, w, stats)
        return y.view(x.shape)

    @staticmethod
    def backward(ctx, dy):
        x2, w, stats = ctx.saved_tensors
        x2, stats = vectors_of(x2), stats.contiguous()  # a saved-tensor hook may answer with other strides
        M, D = x2.shape
        dy2, gain = vectors_of(dy.reshape(-1, D)), vectors_of(w)
        dx = torch.empty_like(x2)
        dw = torch.empty_like(w, memory_format=torch.contiguous_format)
        db = torch.empty_like(dw)
        blocks = lib().tb_layernorm_bwd_blocks(M)
        scratch = torch.empty(blocks * 2 * D, dtype=torch.float32, device=x2.device)
        check_rc(lib().tb_layernorm_bwd(dy2.data_ptr(), x2.data_ptr(), gain.data_ptr(), stats.data_ptr(), stats.data_ptr() + 4 * M, dx.data_ptr(),
                                        dw.data_ptr(), db.data_ptr(), scratch.data_ptr(), M, D, stream(x2)), "layernorm backward")
        return dx.view(dy.shape), dw, db, None


def layer_norm(x, weight, bias, eps=1e-5):
    native = direct(x, weight, bias)
    if native is not None:
        return native.layer_norm(x, weight, bias, eps)
    return run(_LayerNorm, x, weight, bias, eps)


class _ResidualLayerNorm(torch.autograd.Function):
    """(x, LayerNorm(x)): the input is handed through for the residual connection, so that backward receives
    both gradients of x -- the residual branch's and the normalised branch's -- and the LayerNorm backward kernel
    sums them in fp32 while it writes dx, instead of autograd adding them in a pass of its own."""

    @staticmethod
    def forward(ctx, x, w, b, eps):
        need_bf16(x, w, b)
        need(x.dim() > 0 and w.numel() == x.shape[-1] == b.numel(), "layer_norm takes a weight and a bias with one value per column")
        x2 = vectors_of(x.reshape(-1, x.shape[-1]))
        gain, shift = vectors_of(w), vectors_of(b)
        M, D = x2.shape
        y = torch.empty_like(x2)
        stats = torch.empty(2, M, dtype=torch.float32, device=x.device)  # the rows' mean and 1 / std
        check_rc(lib().tb_layernorm_fwd(x2.data_ptr(), gain.data_ptr(), shift.data_ptr(), y.data_ptr(), stats.data_ptr(), stats.data_ptr() + 4 * M,
                                        M, D, eps, stream(x)), "layernorm forward")
        ctx.save_for_backward(x2, w, stats)
        return x.view_as(x), y.view(x.shape)

    @staticmethod
    def backward(ctx, dres, dy):
        x2, w, stats = ctx.saved_tensors
        x2, stats = vectors_of(x2), stats.contiguous()  # a saved-tensor hook may answer with other strides
        M, D = x2.shape
        if dy is None:
            return dres, None, None, None
        dy2, gain = vectors_of(dy.reshape(-1, D)), vectors_of(w)
        add = None if dres is None else vectors_of(dres.reshape(-1, D))
        dx = torch.empty_like(x2)
        dw = torch.empty_like(w, memory_format=torch.contiguous_format)
        db = torch.empty_like(dw)
        blocks = lib().tb_layernorm_bwd_blocks(M)
        scratch = torch.empty(blocks * 2 * D, dtype=torch.float32, device=x2.device)
        check_rc(lib().tb_layernorm_bwd_add(dy2.data_ptr(), x2.data_ptr(), gain.data_ptr(), stats.data_ptr(), stats.data_ptr() + 4 * M,
                                            None if add is None else add.data_ptr(), dx.data_ptr(), dw.data_ptr(), db.data_ptr(),
                                            scratch.data_ptr(), M, D, stream(x2)), "layernorm backward")
        return dx.view(dy.shape), dw, db, None


def residual_layer_norm(x, weight, bias, eps=1e-5):
    """Returns (x, LayerNorm(x)); use the returned x for the residual connection."""
    native = direct(x, weight, bias)
    if native is not None:
        return native.residual_layer_norm(x, weight, bias, eps)
    return run(_ResidualLayerNorm, x, weight, bias, eps)
