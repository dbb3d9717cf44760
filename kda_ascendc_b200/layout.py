"""Chunk-major layouts.

``pack_tokens`` / ``unpack_tokens`` keep the helper names and meaning of the reference
(``python/kda_ascendc_v1/layout.py:17-32``): the leading index of a packed tensor is
``c = (b * H + h) * NT + chunk``.  ``unpack_records`` decodes the K1 -> K2 workspace of
this build (record layout: ``csrc/kda_common.cuh``) back into plain tensors in the
public ``[B, T, H, *]`` layout for stage-wise checks.
"""
from __future__ import annotations

import torch

CHUNK = 16
D = 128
REC_BYTES = 26112
WS_HEADER_BYTES = 256
REC_W, REC_QG, REC_KGH, REC_KGL, REC_AQK, REC_AQL, REC_DEC = 0, 2048, 8192, 12288, 16384, 16640, 17408
REC_XBH, REC_XBL, REC_DEC2, REC_V, REC_USED_BYTES = 17920, 18432, 18944, 19456, 23552
REC_HALF = 4096   # from a 64-column half of w / qg to the other


def pack_tokens(x: torch.Tensor, chunk: int = CHUNK) -> torch.Tensor:
    """``[B, T, H, D]`` -> ``[B*H*(T//chunk), chunk, D]`` (contiguous)."""
    if x.dim() != 4:
        raise ValueError("pack_tokens expects a 4-D [B, T, H, D] tensor")
    b, t, h, d = x.shape
    if t % chunk:
        raise ValueError(f"T={t} is not a multiple of chunk={chunk}")
    return x.view(b, t // chunk, chunk, h, d).permute(0, 3, 1, 2, 4).reshape(-1, chunk, d).contiguous()


def unpack_tokens(x: torch.Tensor, b: int, t: int, h: int, chunk: int = CHUNK) -> torch.Tensor:
    """Inverse of :func:`pack_tokens`."""
    d = x.shape[-1]
    return x.view(b, h, t // chunk, chunk, d).permute(0, 2, 3, 1, 4).reshape(b, t, h, d).contiguous()


def _swizzle_index(device) -> torch.Tensor:
    """Position (in bf16 elements) of element (r, c) inside a w or qg tile, its two 64-column halves back to back."""
    r = torch.arange(CHUNK, device=device)[:, None]
    c = torch.arange(D, device=device)[None, :]
    return ((c >> 6) * 1024 + r * 64 + ((((c >> 3) & 7) ^ (r & 7)) << 3) + (c & 7)).reshape(-1)


def _wq_index(device) -> torch.Tensor:
    """Byte offset of element (r, c) of w or qg inside a record, relative to its part of the first half."""
    at = 2 * _swizzle_index(device).view(CHUNK, D)
    return at + (at >= 2048) * (REC_HALF - 2048)


def _kg_index(device) -> torch.Tensor:
    """Byte offset of element (token, k) inside a transposed kg tile."""
    t = torch.arange(CHUNK, device=device)[:, None]
    k = torch.arange(D, device=device)[None, :]
    return (t >> 3) * 2048 + k * 16 + ((t & 7) << 1)


def _aq_index(device) -> torch.Tensor:
    """Byte offset of element (i, j) of Aqk's hi (or lo) part."""
    i = torch.arange(CHUNK, device=device)[:, None]
    j = torch.arange(CHUNK, device=device)[None, :]
    return (j >> 3) * 512 + i * 16 + ((j & 7) << 1)


def _xb_index(device) -> torch.Tensor:
    """Byte offset of element (i, j) of the hi (or lo) part of X diag(beta)."""
    i = torch.arange(CHUNK, device=device)[:, None]
    j = torch.arange(CHUNK, device=device)[None, :]
    return (j >> 3) * 256 + i * 16 + ((j & 7) << 1)


def _dec2_index(device) -> torch.Tensor:
    """Position (in fp32 elements) of element k of the decay's second copy."""
    k = torch.arange(D, device=device)
    return (k >> 5) * 32 + (k & 7) * 4 + ((k >> 3) & 3)


def _u_index(device) -> torch.Tensor:
    """Position (in fp32 elements) of u[tok][v] in the accumulator fragments of an 8-row K2: [column tile][lane][4]."""
    tok = torch.arange(CHUNK, device=device)[:, None]
    v = torch.arange(D, device=device)[None, :]
    tile, vr = v // 8, v % 8
    lane = (tok % 8) * 4 + vr // 2
    e = (tok // 8) * 2 + vr % 2
    return ((tile * 32 + lane) * 4 + e).reshape(-1)


def unpack_records(workspace: torch.Tensor, B: int, T: int, H: int) -> dict:
    """Decode the chunk records of a finished K1 pass.

    Returns ``w, qg`` (bf16), ``kg, u`` (fp32; kg = hi + lo, u = X diag(beta) v of what the record holds), ``Aqk`` (fp32 = hi + lo, ``[B,T,H,16]``)
    in the public token layout (rows past ``T`` dropped) and ``dec`` fp32 ``[B,H,NT,128]``.
    """
    nt = (T + CHUNK - 1) // CHUNK
    c = B * H * nt
    rec = workspace[WS_HEADER_BYTES:WS_HEADER_BYTES + c * REC_BYTES].view(c, REC_BYTES)
    dev = workspace.device
    half_words = rec.view(torch.bfloat16)   # [c, REC_BYTES / 2]

    def elements(off, index):
        return half_words[:, ((off + index) >> 1).reshape(-1)].view(c, *index.shape)

    def to_public(x):  # [c, 16, n] -> [B, T, H, n]
        n = x.shape[-1]
        y = x.view(B, H, nt, CHUNK, n).permute(0, 2, 3, 1, 4).reshape(B, nt * CHUNK, H, n)
        return y[:, :T].contiguous()

    wq, kg, aq, xb = _wq_index(dev), _kg_index(dev), _aq_index(dev), _xb_index(dev)
    v = elements(REC_V, 2 * _swizzle_index(dev).view(CHUNK, D)).float()
    u = (elements(REC_XBH, xb).double() + elements(REC_XBL, xb).double()) @ v.double()
    aqk = elements(REC_AQK, aq).float() + elements(REC_AQL, aq).float()
    dec = rec[:, REC_DEC:REC_DEC + 512].contiguous().view(torch.float32).view(B, H, nt, D)
    return dict(w=to_public(-elements(REC_W, wq)), qg=to_public(elements(REC_QG, wq)),
                kg=to_public(elements(REC_KGH, kg).float() + elements(REC_KGL, kg).float()),
                u=to_public(u.float()), Aqk=to_public(aqk), dec=dec)
