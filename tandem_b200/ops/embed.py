"""Token + position embedding in one gather kernel; backward scatters token
gradients with fp32 atomics and sums position gradients over the batch in a
fixed order (tandem_b200/cuda/layers.cu)."""

import torch

from ._lib import check_rc, direct, lib, need, need_bf16, need_ids, run, stream, vectors_of


class _Embedding(torch.autograd.Function):
    @staticmethod
    def forward(ctx, idx, tok, pos):
        need_bf16(tok, pos)
        B, T = idx.shape
        need_ids(idx, tok)
        need(tok.dim() == 2 and pos.dim() == 2 and tok.shape[1] == pos.shape[1], "embedding takes two 2-D tables of one width")
        need(T <= pos.shape[0], "more positions than the table has rows")
        D = tok.shape[1]
        idx, tokens, positions = idx.contiguous(), vectors_of(tok), vectors_of(pos)
        out = torch.empty(B, T, D, dtype=torch.bfloat16, device=tok.device)
        check_rc(lib().tb_embed_fwd(idx.data_ptr(), tokens.data_ptr(), positions.data_ptr(), out.data_ptr(), B * T, T, D, stream(tok)),
                 "embedding forward")
        ctx.save_for_backward(idx)
        ctx.shapes = (tok.shape, pos.shape)
        return out

    @staticmethod
    def backward(ctx, dy):
        idx = ctx.saved_tensors[0].contiguous()
        (V, D), (S, _) = ctx.shapes
        B, T = idx.shape
        dy = vectors_of(dy)
        dtok32 = torch.zeros(V, D, dtype=torch.float32, device=dy.device)
        dtok = torch.empty(V, D, dtype=torch.bfloat16, device=dy.device)
        dpos = torch.zeros(S, D, dtype=torch.bfloat16, device=dy.device)
        check_rc(lib().tb_embed_bwd(idx.data_ptr(), dy.data_ptr(), dtok32.data_ptr(), dtok.data_ptr(), dpos.data_ptr(), B, T, D, V,
                                    stream(dy)), "embedding backward")
        return None, dtok, dpos


def embedding(idx, tok, pos):
    native = direct(idx, tok, pos)
    if native is not None:
        return native.embedding(idx, tok, pos)
    return run(_Embedding, idx, tok, pos)
