"""Operator layer: quantised operand containers and the fused operators, mirroring the reference's L6 surface.

Reference counterparts (paths relative to the reference checkout):
    ActBuf / act_buf / MXW            infer-opt/round13_mxfp8_full/impl/mx13.py:53-84
    ln_mx8 / quant_rows / gelu_quant  infer-opt/round13_mxfp8_full/impl/mx13.cu:299-330
    lnq / quantx                      infer-opt/round14_fp4_full/impl/lnq14.cu:158-188
    ln_bf16                           infer-opt/round14_fp4_full/impl/ln14.cu:67
    FQ / Site / Calib                 infer-opt/round14_fp4_full/impl/fp4util.py:47-77

Every operator launches on torch's current CUDA stream through the C-ABI, never synchronises and never
falls back to another implementation: a missing library or a failed launch raises KfError.
torch is used for device memory and streams only.  The argument checks, the output allocation and the call itself are native
(csrc/host/kf_host.cpp): in Python they took 12 to 16 us per operator, longer than most kernels of a small model.
"""
from __future__ import annotations

from typing import Optional

import torch

from . import _lib
from ._lib import KF_DT, KF_FMT, KF_G_GELU, KF_Q_GELU, KF_Q_RECIP_DIV, KF_Q_ROUND_BF16, KfError, check

VEC = {"mx8": 32, "nv4": 16, "mx4": 32}

# Launch accounting used by the benchmark: LAUNCHES counts every kernel launched through this module; when TIMING is
# a dict every launch is bracketed by CUDA events on the launching stream under its kernel-class name and BYTES
# accumulates the algorithmic bytes of the memory-bound classes.
LAUNCHES = 0
TIMING = None
BYTES: dict = {}


class _NativeHost:
    """Stands in for the native operator module until the first operator is called, so that this module imports without it."""

    def __getattr__(self, name):
        global _h
        _h = _lib.host()
        return getattr(_h, name)


_h = _NativeHost()


def _timed(name: str, fn, args: tuple, nbytes: int = 0):
    """fn(*args) between two CUDA events, under the name of its kernel class (TIMING is a dict)."""
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    r = fn(*args)
    e1.record()
    TIMING.setdefault(name, []).append((e0, e1))
    if nbytes:
        BYTES[name] = BYTES.get(name, 0) + nbytes
    return r


def _run(name: str, call) -> None:
    """A launch through the ctypes binding (the operators that are called once per frame)."""
    global LAUNCHES
    LAUNCHES += 1
    check(call() if TIMING is None else _timed(name, call, ()), name)


_DT = {torch.float32: KF_DT["f32"], torch.bfloat16: KF_DT["bf16"], torch.float16: KF_DT["f16"]}


def pad128(n: int) -> int:
    return -(-n // 128) * 128


def sf_bytes(R: int, K: int, fmt: str) -> int:
    n = _lib.lib().kf_sf_bytes(R, K, KF_FMT[fmt])
    if n < 0:
        check(int(n), "kf_sf_bytes")
    return int(n)


def code_cols(K: int, fmt: str) -> int:
    return K if fmt == "mx8" else K // 2


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _ptr(t: Optional[torch.Tensor]) -> int:
    return 0 if t is None else t.data_ptr()


def _need_cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise KfError("operands must live on a CUDA device (there is no CPU path)")


class ActBuf:
    """Quantised [M, K] operand: codes q (uint8, [M, K] for mx8, [M, K/2] packed nibbles for nv4 / mx4), blocked
    scales sf (uint8, [ceil(M/128), K/(4 vec), 32, 4, 4] flattened) and, for nv4, the fp32 per-tensor scale ts [1]."""

    __slots__ = ("M", "K", "fmt", "q", "sf", "ts")

    def __init__(self, M: int, K: int, fmt: str = "mx8", device="cuda", ts: Optional[torch.Tensor] = None):
        self.M, self.K, self.fmt = M, K, fmt
        self.q = torch.empty(M, code_cols(K, fmt), dtype=torch.uint8, device=device)
        self.sf = torch.zeros(sf_bytes(M, K, fmt), dtype=torch.uint8, device=device)   # padded rows stay zero
        self.ts = ts if ts is not None else (torch.ones(1, dtype=torch.float32, device=device) if fmt == "nv4" else None)


FQ = ActBuf   # the FP4 stacks call the same container FQ (fp4util.py:54-58)

_POOL: dict = {}


def act_buf(M: int, K: int, fmt: str = "mx8", device="cuda", slot: int = 0) -> ActBuf:
    """persistent operand buffer shared by every layer of one shape (the stream is sequential)."""
    key = (M, K, fmt, slot, str(device))
    if key not in _POOL:
        _POOL[key] = ActBuf(M, K, fmt, device)
    return _POOL[key]


def _flags(gelu=False, round_bf16=False, recip_div=False) -> int:
    return (KF_Q_GELU if gelu else 0) | (KF_Q_ROUND_BF16 if round_bf16 else 0) | (KF_Q_RECIP_DIV if recip_div else 0)


def quant_rows(x: torch.Tensor, out: ActBuf, *, bias: Optional[torch.Tensor] = None, gelu: bool = False,
               round_bf16: bool = False, recip_div: bool = False) -> ActBuf:
    """x [M, K] f32 | bf16 | f16 (last dim contiguous) -> out (codes + blocked scales), format out.fmt.
    gelu=True applies gelu_erf(x + bias) first (the reference's gelu_quant)."""
    global LAUNCHES
    LAUNCHES += 1
    args = (x, out, bias, _flags(gelu, round_bf16, recip_div))
    if TIMING is None:
        return _h.quant_rows(*args)
    return _timed("quant_rows", _h.quant_rows, args, x.numel() * x.element_size() + out.q.numel() + out.sf.numel())


def gelu_quant(y: torch.Tensor, bias: torch.Tensor, out: ActBuf, **kw) -> ActBuf:
    return quant_rows(y, out, bias=bias, gelu=True, **kw)


def quantx(x: torch.Tensor, out: ActBuf, **kw) -> ActBuf:
    return quant_rows(x, out, **kw)


def ln_quant(x: torch.Tensor, w: torch.Tensor, b: torch.Tensor, eps: float, out: ActBuf, *, round_bf16: bool = False,
             recip_div: bool = False, y_dbg: Optional[torch.Tensor] = None, static_affine: bool = False) -> ActBuf:
    """LayerNorm of the fp32 (or bf16) stream x [..., d] fused with quantisation into out (ln_mx8 / lnq).
    static_affine=True promises that every write of w and b was complete before the launch in front of this one began its work:
    they are then read before that launch has ended."""
    global LAUNCHES
    LAUNCHES += 1
    args = (x, w, b, eps, out, _flags(False, round_bf16, recip_div) | (_lib.KF_Q_STATIC_AFFINE if static_affine else 0), y_dbg)
    if TIMING is None:
        return _h.ln_quant(*args)
    return _timed("ln_quant", _h.ln_quant, args, x.numel() * x.element_size() + out.q.numel() + out.sf.numel())


def ln_mx8(x, w, b, out: ActBuf, eps: float, **kw) -> ActBuf:
    return ln_quant(x, w, b, eps, out, **kw)


def lnq(x, w, b, eps: float, out: ActBuf, **kw) -> ActBuf:
    return ln_quant(x, w, b, eps, out, **kw)


def ln_rows(x: torch.Tensor, w: torch.Tensor, b: torch.Tensor, eps: float, dtype=torch.bfloat16) -> torch.Tensor:
    """LayerNorm of fp32 x [..., d] to a bf16 / f16 tensor of the same shape (ln_bf16 / ln16)."""
    global LAUNCHES
    LAUNCHES += 1
    args = (x, w, b, eps, _DT[dtype])
    return _h.ln_rows(*args) if TIMING is None else _timed("ln_rows", _h.ln_rows, args)


ln_bf16 = ln_rows


def amax_scale(x: torch.Tensor, ts: torch.Tensor, ws: torch.Tensor, *, factor: float = 1.0 / 2688.0, gelu: bool = False) -> torch.Tensor:
    """ts [1] = factor * max|v| (1 where that is zero or NaN), v = x [M, K] or gelu_erf(x), in one launch and without a host sync: the
    dynamic per-tensor scale of an NVFP4 operand.  ws: int32 [2], zero before the first use (a call leaves it zero)."""
    global LAUNCHES
    LAUNCHES += 1
    args = (x, KF_Q_GELU if gelu else 0, factor, ts, ws)
    return _h.amax_scale(*args) if TIMING is None else _timed("amax_scale", _h.amax_scale, args)


def ln_amax_scale(x: torch.Tensor, w: torch.Tensor, b: torch.Tensor, eps: float, ts: torch.Tensor, ws: torch.Tensor, *, factor: float = 1.0 / 2688.0) -> torch.Tensor:
    """amax_scale of the bf16-rounded LayerNorm of f32 | bf16 x [..., d], which is not written anywhere."""
    global LAUNCHES
    LAUNCHES += 1
    args = (x, w, b, eps, factor, ts, ws)
    return _h.ln_amax_scale(*args) if TIMING is None else _timed("amax_scale", _h.ln_amax_scale, args)


# ------------------------------------------------------------------------------------------------ weights and GEMMs
def set_pdl(on: Optional[bool]) -> None:
    """Programmatic dependent launch: True = every launch, False = none (plain stream order), None = launches over few rows, which is how
    the package starts; results are the same in all three.  Counterpart: set_pdl (infer-opt/round13_mxfp8_full/impl/mx13.cu:282)."""
    check(_lib.lib().kf_set_pdl(_lib.KF_PDL["auto" if on is None else "all" if on else "off"]), "kf_set_pdl")


def check_device_error() -> None:
    """synchronises and raises if a kernel's bounded wait ran out (no reference counterpart)."""
    check(_lib.lib().kf_check_device_error(), "kf_check_device_error")


def settled(q: torch.Tensor, sf: Optional[torch.Tensor] = None) -> Optional[tuple]:
    """Waits until the writes of these tensors on the current stream are complete; -> (q, sf, sum of their version counters), or None under
    graph capture and for inference tensors (which have no counter)."""
    ts = [t for t in (q, sf) if t is not None]
    if torch.cuda.is_current_stream_capturing() or any(t.is_inference() for t in ts):
        return None
    torch.cuda.current_stream(q.device).synchronize()
    return q, sf, sum(t._version for t in ts)


class QWeight:
    """Weight [N, K] (nn.Linear layout) quantised once along K with 1-D block scales; fmt "bf16" keeps it in bf16.
    nv4: exact per-tensor scale ts = amax/(6*448) computed once on the host cores (IEEE division).
    Counterparts: MXW (infer-opt/round13_mxfp8_full/impl/mx13.py:74-84), Lin / FP4Linear weights
    (infer-opt/round14_fp4_full/impl/stack14b.py:55-66, fp4util.py:114-131).

    The constructor waits for the quantisation (not under graph capture): a GEMM may then request the weights ahead of its
    predecessor's end, as long as nothing has written q or sf since, by their version counters, or put others in their place."""

    def __setattr__(self, name, value):
        if name in ("q", "sf"):
            super().__setattr__("settled", None)       # also: the tensors of the past are not held
        super().__setattr__(name, value)

    def __getstate__(self):
        return {**self.__dict__, "settled": None}          # the tensors of a copy have been written since

    def __init__(self, W: torch.Tensor, fmt: str, ts: Optional[torch.Tensor] = None):
        _need_cuda(W)
        self.N, self.K = W.shape
        self.fmt = fmt
        if fmt == "bf16":
            self.q = W.to(torch.bfloat16).contiguous()
            self.sf = None
            self.ts = None
            self.settled = settled(self.q)
            return
        Wf = W.float().contiguous()
        buf = ActBuf(self.N, self.K, fmt, device=W.device)
        if fmt == "nv4":
            if ts is None:
                import numpy as np

                amax = np.float32(Wf.abs().amax().item())
                ts = torch.tensor([amax / np.float32(2688.0) if amax > 0 else 1.0], dtype=torch.float32)
            buf.ts.copy_(ts.reshape(1))
        quant_rows(Wf, buf)
        self.q, self.sf, self.ts = buf.q, buf.sf, buf.ts
        self.settled = settled(self.q, self.sf)


MXW = QWeight


def gemm_plain(a, W: QWeight, bias=None, *, gelu: bool = False, out_dtype=torch.bfloat16, out: Optional[torch.Tensor] = None,
               tag: str = "block", pre_round: bool = False) -> torch.Tensor:
    """[M, N] = act(a @ W^T (* ts) + bias) in bf16 / f16 / f32 (mm, gemm_plain, fwd_bias, fwd_gelu, fwd_plain)."""
    global LAUNCHES
    LAUNCHES += 1
    args = (a, W, bias, out, _DT[out_dtype], (KF_G_GELU if gelu else 0) | (_lib.KF_G_PRE_ROUND_BF16 if pre_round else 0))
    return _h.gemm_plain(*args) if TIMING is None else _timed(f"gemm_{tag}_{W.fmt}", _h.gemm_plain, args)


mm = gemm_plain


def bmm_nt(a: torch.Tensor, w: torch.Tensor, out: Optional[torch.Tensor] = None, tag: str = "mask") -> torch.Tensor:
    """out[b] = a[b] @ w[b]^T for bf16 a [B, Q, K] and w [B, P, K] in one launch (P a multiple of 128): the mask product
    torch.bmm(h, u.transpose(1, 2)) of the head (infer-opt/round11_attn_tier0/impl/head11.py:95).  Bit-identical to B
    gemm_plain calls; one launch fills the SMs where a single image leaves a partial round of tiles."""
    global LAUNCHES
    LAUNCHES += 1
    args = (a, w, out)
    return _h.bmm_nt(*args) if TIMING is None else _timed(f"gemm_{tag}_bf16", _h.bmm_nt, args)


def gemm_res(a, W: QWeight, bias, gamma, res: torch.Tensor, out: Optional[torch.Tensor] = None, row_map=None) -> torch.Tensor:
    """fp32 [M, N] = res + gamma * (a @ W^T (* ts) + bias)   (proj / fc2; gemm_res, fwd_res).
    row_map = (group, stride, offset): row m of the result goes to row (m // group) * stride + offset + m % group of `out`
    (a longer token stream: the rows of each image land behind `offset` rows that are filled separately); not in place."""
    global LAUNCHES
    LAUNCHES += 1
    args = (a, W, bias, gamma, res, out, row_map)
    return _h.gemm_res(*args) if TIMING is None else _timed(f"gemm_block_{W.fmt}", _h.gemm_res, args)


def broadcast_rows(src: torch.Tensor, dst: torch.Tensor, row_offset: int) -> torch.Tensor:
    """dst[b, row_offset : row_offset + R, :] = src [R, d] for every image b of the fp32 token stream dst [B, Ntok, d]."""
    global LAUNCHES
    LAUNCHES += 1
    args = (src, dst, row_offset)
    return _h.broadcast_rows(*args) if TIMING is None else _timed("broadcast_rows", _h.broadcast_rows, args)


def rope_tables_are_half(sin: torch.Tensor, cos: torch.Tensor) -> bool:
    """True when columns 32..63 of both tables repeat columns 0..31 (the axial tables of DINOv3: the angle vector concatenated
    with itself).  A host-side check (it synchronises): call it once when the tables are built, not per launch."""
    return bool(torch.equal(sin[:, :32], sin[:, 32:]) and torch.equal(cos[:, :32], cos[:, 32:]))


def qkv_rope(a, W: QWeight, bias, sin, cos, Ntok: int, prefix: int, H: int, out_dtype=torch.bfloat16, half_tables: bool = False) -> torch.Tensor:
    """a [M=B*Ntok, d] -> physical [3, B, Ntok, H, 64] (bias + RoPE in fp32 on q and k of tokens >= prefix).
    half_tables=True promises rope_tables_are_half(sin, cos): the kernel then keeps a tile's table rows in shared memory."""
    global LAUNCHES
    LAUNCHES += 1
    args = (a, W, bias, sin, cos, Ntok, prefix, H, _DT[out_dtype], _lib.KF_G_ROPE_HALF if half_tables else 0)
    return _h.qkv_rope(*args) if TIMING is None else _timed(f"gemm_block_{W.fmt}", _h.qkv_rope, args)


def gemm_gelu_q(a, W: QWeight, bias, out: ActBuf, *, round_bf16: bool = False, recip_div: bool = False, fast_nv4: bool = False,
                y_dbg: Optional[torch.Tensor] = None) -> ActBuf:
    """out = quantise(gelu(a @ W^T (* ts) + bias)) in out.fmt: fc1 writes fc2's operand and blocked scales directly.
    The quantisation follows the bit specification (IEEE divisions); fast_nv4=True selects approximate reciprocals for an
    nv4 output.  y_dbg (fp32 [M, N], optional) receives the values that were quantised."""
    global LAUNCHES
    LAUNCHES += 1
    args = (a, W, bias, out, _flags(False, round_bf16, recip_div) | (_lib.KF_Q_FAST_NV4 if fast_nv4 else 0), y_dbg)
    return _h.gemm_gelu_q(*args) if TIMING is None else _timed(f"gemm_block_{W.fmt}", _h.gemm_gelu_q, args)


# ------------------------------------------------------------------------------------------------ attention
def attn_fwd(qkv: torch.Tensor, pre: float = 1.0, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """qkv contiguous [3, B, N, H, 64] bf16 | f16 (RoPE applied) -> O [B, N, H*64] of the same dtype.
    Counterpart: attn16_fwd(qkv, kind, pre) (infer-opt/round12_lowp_stack/impl/attn16o.cu:389-404)."""
    global LAUNCHES
    LAUNCHES += 1
    args = (qkv, pre, out)
    return _h.attn_fwd(*args) if TIMING is None else _timed("attn_fwd", _h.attn_fwd, args)


attn16_fwd = attn_fwd


def attn_fwd_quant(qkv: torch.Tensor, out: ActBuf, pre: float = 1.0, recip_div: bool = False) -> ActBuf:
    """attention forward whose output is written directly as the quantised [B*N, H*64] operand `out` (codes + blocked
    scales; out.ts is the static nv4 scale): attn16_fwd + quant_rows in one kernel."""
    global LAUNCHES
    LAUNCHES += 1
    args = (qkv, out, pre, KF_Q_RECIP_DIV if recip_div else 0)
    return _h.attn_fwd_quant(*args) if TIMING is None else _timed("attn_fwd", _h.attn_fwd_quant, args)


# ------------------------------------------------------------------------------------------------ patch embed / head / pre / post
def gemm_tokens(a: torch.Tensor, W: QWeight, bias, out: torch.Tensor, rows_per_image: int, tokens_per_image: int, row_offset: int,
                round_bf16: bool = False) -> torch.Tensor:
    """patch-embed GEMM: a bf16 [B*P, K] @ W^T + bias written as fp32 rows row_offset.. of every image of the token
    stream out [B, tokens_per_image, N] (counterpart: PatchEmbedGemm, infer-opt/round11_attn_tier0/impl/patch_embed.py:34-53)."""
    global LAUNCHES
    LAUNCHES += 1
    args = (a, W, bias, out, rows_per_image, tokens_per_image, row_offset, _lib.KF_G_ROUND_BF16 if round_bf16 else 0)
    return _h.gemm_tokens(*args) if TIMING is None else _timed("gemm_patch_bf16", _h.gemm_tokens, args)


PATCH_STATIC_MAX_ROWS = 4096


def patch_embed_static(x: torch.Tensor, W: QWeight, bias, out: torch.Tensor, row_offset: int, round_bf16: bool = False) -> torch.Tensor:
    """Patch embedding for callers that must not allocate: x bf16 [B, 3, S, S] -> rows row_offset.. of every image of the fp32
    token stream out [B, tokens_per_image, d], through the library's built-in scratch array instead of an im2col tensor
    (the same bits as gemm_tokens(im2col_patch16(x), ...)).  At most PATCH_STATIC_MAX_ROWS patch rows per call; calls that
    overlap on the GPU race on the shared array; the first call on a device should come before any stream capture."""
    _need_cuda(x, W.q, bias, out)
    if x.dtype != torch.bfloat16 or x.dim() != 4 or x.shape[1] != 3 or x.shape[2] != x.shape[3] or not x.is_contiguous():
        raise KfError("patch_embed_static: x must be contiguous bf16 [B, 3, S, S]")
    if W.fmt != "bf16" or W.K != 768 or out.dtype != torch.float32 or not out.is_contiguous() or out.dim() != 3 or out.shape[2] != W.N:
        raise KfError("patch_embed_static: W must be a bf16 [d, 768] weight and out contiguous fp32 [B, tokens_per_image, d]")
    B, _, S, _ = x.shape
    _run("patch_embed_static", lambda: _lib.lib().kf_patch_embed_static(x.data_ptr(), W.q.data_ptr(), _ptr(bias), out.data_ptr(), B, S, W.N, out.shape[1], row_offset,
                                                                        _lib.KF_G_ROUND_BF16 if round_bf16 else 0, _stream()))
    return out


def im2col_patch16(x: torch.Tensor) -> torch.Tensor:
    """x bf16 [B, 3, S, S] -> bf16 [B*(S/16)^2, 768]."""
    global LAUNCHES
    LAUNCHES += 1
    return _h.im2col_patch16(x) if TIMING is None else _timed("im2col_patch16", _h.im2col_patch16, (x,))


def ln_tail(x: torch.Tensor, w, b, eps: float, Q: int, npre: int, wcls: Optional[torch.Tensor] = None, bcls: Optional[torch.Tensor] = None):
    """final LayerNorm + gather: x fp32 [B, Ntok, d] -> (queries bf16 [B*Q, d], patches bf16 [B*(Ntok-Q-npre), d]), and with
    wcls bf16 [ncls1, d] / bcls fp32 [ncls1] the class logits bf16 [B*Q, ncls1] of the query rows as a third result."""
    global LAUNCHES
    LAUNCHES += 1
    args = (x, w, b, eps, Q, npre, wcls, bcls)
    return _h.ln_tail(*args) if TIMING is None else _timed("ln_tail", _h.ln_tail, args)


def dw_ln(g: torch.Tensor, bias, dww, lnw, lnb, B: int, Hs: int, Ws: int, eps: float, pre_act: bool = False) -> torch.Tensor:
    """ScaleBlock tail: g bf16 [B*Hs*Ws, 4C] -> bf16 [B, 2Hs, 2Ws, C] (dw_ln_launch, head11.py:60-67).
    pre_act=True: g already is bf16(gelu(conv + bias)) (fused into the GEMM epilogue), bias may be None."""
    global LAUNCHES
    LAUNCHES += 1
    args = (g, bias, dww, lnw, lnb, B, Hs, Ws, eps, pre_act)
    return _h.dw_ln(*args) if TIMING is None else _timed("dw_ln", _h.dw_ln, args)


def semantic(mask_logits: torch.Tensor, class_logits: torch.Tensor, want_scores: bool = False):
    """mask_logits bf16 [B, Q, h, w], class_logits bf16 [B, Q, ncls+1] -> (labels uint8 [B, h, w], scores fp32 [B, ncls+1, h, w] | None)."""
    global LAUNCHES
    LAUNCHES += 1
    args = (mask_logits, class_logits, want_scores)
    return _h.semantic(*args) if TIMING is None else _timed("semantic", _h.semantic, args)


IMAGENET_MEAN = (0.485, 0.456, 0.406)
IMAGENET_STD = (0.229, 0.224, 0.225)


def resize_norm(frames: torch.Tensor, size: int, mean=IMAGENET_MEAN, std=IMAGENET_STD, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """frames uint8 [B, Hi, Wi, 3] -> bf16 [B, 3, size, size] (antialiased bilinear + normalisation)."""
    import ctypes as C

    _need_cuda(frames)
    if frames.dtype != torch.uint8 or frames.dim() != 4 or frames.shape[3] != 3 or not frames.is_contiguous():
        raise KfError("resize_norm: frames must be contiguous uint8 [B, H, W, 3]")
    B, Hi, Wi, _ = frames.shape
    if out is None:
        out = torch.empty(B, 3, size, size, dtype=torch.bfloat16, device=frames.device)
    m, s = (C.c_float * 3)(*mean), (C.c_float * 3)(*std)
    _run("resize_norm", lambda: _lib.lib().kf_resize_norm(frames.data_ptr(), out.data_ptr(), B, Hi, Wi, size, m, s, _stream()))
    return out


def tensor_peak_tflops(fmt: str, n: int = 256, iters: int = 4096, reps: int = 5, sf_copies: int = 0) -> float:
    """measured tcgen05 instruction-rate ceiling (TFLOP/s) for operand format fmt at M=128, N=n (best of reps)."""
    import ctypes as C

    fl = C.c_double(0.0)
    L = _lib.lib()
    best = 0.0
    for _ in range(reps + 1):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        check(L.kf_tensor_peak_probe(KF_FMT[fmt], n, iters, sf_copies, C.byref(fl), _stream()), "kf_tensor_peak_probe")
        e1.record()
        e1.synchronize()
        best = max(best, fl.value / (e0.elapsed_time(e1) * 1e-3) / 1e12)
    return best


def smem_fill_rate_gbs(span_bytes: int, stage_bytes: int = 49152, iters: int = 2048, reps: int = 5) -> float:
    """measured rate (GB/s, all SMs together) at which bulk copies fill shared memory from a window of span_bytes of
    global memory that fits L2 (best of reps)."""
    import ctypes as C

    src = torch.empty(span_bytes, dtype=torch.uint8, device="cuda").zero_()
    nb = C.c_double(0.0)
    L = _lib.lib()
    best = 0.0
    for _ in range(reps + 1):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        check(L.kf_fill_rate_probe(src.data_ptr(), span_bytes, stage_bytes, iters, C.byref(nb), _stream()), "kf_fill_rate_probe")
        e1.record()
        e1.synchronize()
        best = max(best, nb.value / (e0.elapsed_time(e1) * 1e-3) / 1e9)
    check_device_error()
    return best
