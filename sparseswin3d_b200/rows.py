"""Row passes around the GEMMs of a block with autograd recording: residual add + LayerNorm, and the
bias gradient of a Linear layer, each forward and backward one pass over the voxel rows (csrc/norm.cu).

torch's own kernels stay for everything these do not cover: other dtypes, mixed dtypes, rows that are not
16-byte multiples, autocast, module hooks, function transforms, forward-mode differentiation, tracing.
Under create_graph the backward is written in differentiable torch operations."""
from __future__ import annotations

import contextvars
from typing import Optional

import torch
import torch.nn as nn
import torch.nn.functional as F

from ._lib import H_ERROR, SswError, check, dtype_code, lib, ptr, stream_ptr

_DTYPES = (torch.float32, torch.bfloat16, torch.float16)

# Rows from which the passes are used while autograd records: below, a training step waits for the host, and an autograd
# function in Python costs it more than torch's own.  One block, forward and backward, 96 channels, with / without:
# residual add + LayerNorm, bf16: 25 000 rows 1136 / 1063 us, 40 000 rows 1125 / 1401; fp32: 1178 / 1156, 1205 / 1626.
ADD_NORM_ROWS = 32768
# Linear, fp32 (the GEMM): 12 000 rows 1128 / 1056 us, 25 000 rows 1178 / 1368, 40 000 rows 1205 / 1922.
LINEAR_ROWS_F32 = 16384
# Wider Linears: (their narrower side, rows).  A stage of two blocks, with / without, on two hosts (what it takes at least is the host's time, 1950 to
# 2300 us with, 1910 to 2050 without): 192 channels, 4096 rows 2016 / 1921 and 1996 / 1927 us, 5000 2108 / 2115 and 1964 / 2109, 7000 2210 / 2674; 384 channels,
# 1500 rows 2233 / 2105, 2000 2287 / 2135 and 1946 / 2131, 2500 2501 / 2606 and 1932 / 2314; 768 channels, 512 rows 2378 / 2101 and 1972 / 1913, 850
# 1983 / 2758, 1024 2164 / 2949 and 1958 / 2875.  96 channels, 12 000 rows 2431 / 2319, 16 384 2141 / 2613.  From these rows on the three products of such a
# Linear are ones that pay (see _gemm_pays).
LINEAR_ROWS_F32_WIDE = ((768, 1024), (384, 2500), (192, 5000))
# Linear, 16 bits (the bias gradient alone), rows at 96 channels: 40 000 rows 1143 / 1125.  A stage of two blocks: 66 000 rows of 96 channels
# 2245 / 2010, 100 000 2141 / 2170, 150 000 2464 / 2814; 150 000 of 48 2111 / 2065.
LINEAR_ROWS_16 = 100000


# The window plan whose error word the GEMMs of a call report to (the strict checks read it), where none is handed over.
_plan = contextvars.ContextVar("plan", default=None)


class reporting:
    """with reporting(plan): time-outs of the GEMMs called here go to the plan's error word."""

    def __init__(self, plan):
        self.plan = plan

    def __enter__(self):
        self.token = _plan.set(self.plan)

    def __exit__(self, *exc):
        _plan.reset(self.token)


def _error_word(plan, device) -> int:
    return ptr(plan.plan) + 4 * (plan.layout.off_header + H_ERROR) if plan is not None and plan.plan.device == device else 0


def unhooked(*modules: nn.Module) -> bool:
    """Calling the module and using its parameters directly are the same thing."""
    g = nn.modules.module
    return not (g._global_forward_hooks or g._global_forward_pre_hooks or g._global_backward_hooks or g._global_backward_pre_hooks
                or any(m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks
                       or "forward" in m.__dict__ or m._compiled_call_impl is not None for m in modules))


def _ordinary_mode() -> bool:
    return not (torch.is_autocast_enabled("cuda") or torch._C._are_functorch_transforms_active()
                or torch.autograd.forward_ad._current_level >= 0 or torch._C._is_tracing() or torch.compiler.is_compiling())


def aligned_rows(*tensors: torch.Tensor) -> bool:
    """[n, C] CUDA rows the kernels take: contiguous, 16-byte aligned, n > 0, C * element size a multiple of 16."""
    return all(type(t) in (torch.Tensor, nn.Parameter) and t.is_cuda and t.device.index == torch.cuda.current_device() and t.dim() == 2
               and t.dtype in _DTYPES and t.is_contiguous() and t.shape[0] > 0
               and (t.shape[1] * t.element_size()) % 16 == 0 and t.data_ptr() % 16 == 0 for t in tensors)


def plain_norm(norm, x: torch.Tensor) -> bool:
    """`norm` is an affine LayerNorm over the rows of `x`, in their dtype, that the kernels reproduce."""
    return (type(norm) is nn.LayerNorm and tuple(norm.normalized_shape) == (x.shape[-1],) and norm.weight is not None
            and norm.bias is not None and norm.weight.shape == norm.bias.shape == norm.normalized_shape and norm.weight.dtype == x.dtype and norm.bias.dtype == x.dtype
            and norm.weight.device == x.device and norm.bias.device == x.device
            and norm.weight.is_contiguous() and norm.bias.is_contiguous()
            and x.shape[-1] * x.element_size() <= 2048 and unhooked(norm) and _ordinary_mode())


def norm_params(norm: nn.LayerNorm):
    """(weight, bias, dtype code) as the kernels read them: in place where the module's type allows."""
    w, b = norm.weight, norm.bias
    if not w.shape == b.shape == norm.normalized_shape:
        raise SswError(f"LayerNorm parameters {tuple(w.shape)} and {tuple(b.shape)} are not of the normalised shape {norm.normalized_shape}")
    if w.dtype != b.dtype or w.dtype not in _DTYPES or not (w.is_contiguous() and b.is_contiguous()):
        w, b = w.detach().float().contiguous(), b.detach().float().contiguous()
    return w, b, dtype_code(w.dtype)


class _AddLayerNorm(torch.autograd.Function):
    """(a + b, LayerNorm(a + b)); b None: (a, LayerNorm(a))."""

    @staticmethod
    def forward(ctx, a, b, weight, bias, eps):
        n, c = a.shape
        s = torch.empty_like(a) if b is not None else a.view_as(a)
        y = torch.empty_like(a)
        code = dtype_code(a.dtype)
        check(lib.ssw_add_layernorm_p(ptr(a), ptr(b), ptr(weight), ptr(bias), code, float(eps), code, n, c,
                                      ptr(s) if b is not None else 0, ptr(y), stream_ptr(a.device)), "ssw_add_layernorm")
        ctx.set_materialize_grads(False)
        ctx.eps, ctx.pair = float(eps), b is not None
        ctx.save_for_backward(s if b is not None else a, weight)
        return s, y

    @staticmethod
    def backward(ctx, ds, dy):
        x, weight = ctx.saved_tensors
        if dy is None:
            return ds, ds if ctx.pair else None, None, None, None
        if torch.is_grad_enabled():  # create_graph: differentiable operations
            xf, g = x.float(), dy.float()
            xc = xf - xf.mean(1, keepdim=True)
            rstd = (xc.square().mean(1, keepdim=True) + ctx.eps).rsqrt()
            xh, wg = xc * rstd, g * weight.float()
            dx = (rstd * (wg - wg.mean(1, keepdim=True) - xh * (wg * xh).mean(1, keepdim=True))).to(x.dtype)
            if ds is not None:
                dx = dx + ds
            return dx, dx if ctx.pair else None, (g * xh).sum(0).to(weight.dtype), g.sum(0).to(weight.dtype), None
        n, c = x.shape
        dy = _rows(dy)
        ds = None if ds is None else _rows(ds)
        dx = torch.empty_like(x)
        dw, db = torch.empty_like(weight), torch.empty_like(weight)
        ws = torch.empty(int(lib.ssw_layernorm_bwd_workspace_floats(n, c)), dtype=torch.float32, device=x.device)
        code = dtype_code(x.dtype)
        check(lib.ssw_layernorm_bwd(ptr(x), ptr(dy), ptr(ds), ptr(weight), code, ctx.eps, code, n, c, ptr(dx), ptr(dw), ptr(db), ptr(ws),
                                    stream_ptr(x.device)), "ssw_layernorm_bwd")
        return dx, dx if ctx.pair else None, dw, db, None


def _rows(g: torch.Tensor) -> torch.Tensor:
    g = g.contiguous()
    return g if g.data_ptr() % 16 == 0 else g.clone()


def add_layer_norm(a: torch.Tensor, b: Optional[torch.Tensor], norm: nn.LayerNorm):
    """(a + b, norm(a + b)) with autograd; the caller has checked `aligned_rows` and `plain_norm`."""
    return _AddLayerNorm.apply(a, b, norm.weight, norm.bias, norm.eps)


def col_sum(g: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    """Sum over the rows of g [n, C] (fp32 accumulation), in `dtype`."""
    n, c = g.shape
    out = torch.empty(c, dtype=dtype, device=g.device)
    ws = torch.empty(int(lib.ssw_col_sum_workspace_floats(n, c)), dtype=torch.float32, device=g.device)
    check(lib.ssw_col_sum(ptr(g), dtype_code(g.dtype), n, c, ptr(out), dtype_code(dtype), ptr(ws), stream_ptr(g.device)), "ssw_col_sum")
    return out


_fp32_precision = torch._C._get_fp32_precision_getter  # torch.backends.cuda.matmul.fp32_precision


def _gemm_ready(x: torch.Tensor, weight: torch.Tensor, first: int = 0) -> bool:
    """x [M, K] and weight [N, K] (first = 1: g [M, N] and x [M, K]) suit the fp32 GEMM, and torch is not told to use TF32 for
    such products."""
    return (x.dtype == torch.float32 and weight.dtype == torch.float32 and x.is_contiguous() and weight.is_contiguous()
            and x.data_ptr() % 16 == 0 and weight.data_ptr() % 16 == 0 and (x if first else weight).shape[first] % 4 == 0
            and weight.shape[1] % 4 == 0
            and _fp32_precision("cuda", "matmul") in ("ieee", "none"))


def _gemm_pays(m: int, n: int, k: int) -> bool:
    """From where the fp32 GEMM is taken for a product.  The library's splits K where few tiles of results leave the chip idle; the line lies where the two met
    while a tile here took 1.5 times as long as it does now.  Above it this one is faster at every pair measured; below it so too from 128 rows on, by up to
    1.7 times, and slower with a few rows of a long sum.  With bias, (N, K): rows library / own in us, * below the line.  (96, 96): *128 5.9 / 4.3,
    *1000 6.1 / 4.3, 2500 7.1 / 4.5; (576, 192): *128 7.5 / 6.1, 512 9.0 / 6.2; (96, 384): *2500 12 / 9, 5000 18 / 10; (192, 768): *64 15 / 14, *1500 19 / 15,
    2500 26 / 16; (384, 1536): *64 19 / 26, *512 32 / 27, *1000 44 / 29, 1500 45 / 29; (768, 3072): *1 5 / 50, *256 59 / 50, 512 81 / 55."""
    return m * n >= 1024 * min(k, 384)


def _gemm(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], plan=None) -> torch.Tensor:
    (m, k), n = x.shape, weight.shape[0]
    out = torch.empty((m, n), dtype=torch.float32, device=x.device)
    check(lib.ssw_gemm_f32(ptr(x), ptr(weight), ptr(bias), ptr(out), m, n, k, _error_word(plan, x.device), stream_ptr(x.device)),
          "ssw_gemm_f32")
    return out


def _gemm_tn(g: torch.Tensor, x: torch.Tensor, plan=None) -> torch.Tensor:
    (m, n), k = g.shape, x.shape[1]
    out = torch.empty((n, k), dtype=torch.float32, device=x.device)
    ws = torch.empty(int(lib.ssw_gemm_f32_tn_workspace_floats(m, n, k)), dtype=torch.float32, device=x.device)
    check(lib.ssw_gemm_f32_tn(ptr(g), ptr(x), ptr(out), m, n, k, ptr(ws), _error_word(plan, x.device), stream_ptr(x.device)),
          "ssw_gemm_f32_tn")
    return out


def _bias_ready(bias: Optional[torch.Tensor], n: int) -> bool:
    """The kernels read `n` consecutive values (fp32: in 16-byte pieces); a Linear takes any bias that broadcasts."""
    return bias is None or (bias.is_contiguous() and bias.dim() == 1 and bias.shape[0] == n
                            and (bias.data_ptr() % 16 == 0 or bias.dtype != torch.float32))


def _affine(x, weight, bias, plan=None):
    n, k = weight.shape
    if _gemm_pays(x.shape[0], n, k) and _gemm_ready(x, weight) and _bias_ready(bias, n):
        return _gemm(x, weight, bias, plan)
    return F.linear(x, weight, bias)


class _Linear(torch.autograd.Function):
    """F.linear; in fp32 the product and both gradients are the tensor-core GEMM, and the backward sums the bias gradient
    in one pass over the rows."""

    @staticmethod
    def forward(ctx, x, weight, bias, plan=None):
        ctx.save_for_backward(x, weight)
        ctx.plan = plan
        return _affine(x, weight, bias, plan)

    @staticmethod
    def backward(ctx, g):
        x, weight = ctx.saved_tensors
        need = ctx.needs_input_grad
        if torch.is_grad_enabled():  # create_graph: differentiable operations
            return (g @ weight if need[0] else None, g.t() @ x if need[1] else None, g.sum(0) if need[2] else None, None)
        g = _rows(g)
        gx = gw = gb = None
        if need[0]:
            # (no question of _gemm_pays: with 16 384 rows the own product is the faster one too where few input channels say otherwise, 16 of them
            # and 384 outputs 11 us for 14, 20 and 3072 59 for 98; and with fewer rows the lines above are ones from which it pays)
            wt = weight.t()
            if g.dtype == torch.float32 and weight.shape[1] % 4 == 0:
                wt = wt.contiguous()
            gx = _gemm(g, wt, None, ctx.plan) if _gemm_ready(g, wt) else g @ weight
        if need[1]:
            gw = _gemm_tn(g, x, ctx.plan) if _gemm_ready(g, x, 1) else g.t() @ x
        if need[2]:
            gb = col_sum(g, g.dtype)
        return gx, gw, gb, None


def _own_linear(module: nn.Module, x: torch.Tensor):
    """(weight, bias) of a Linear whose call the passes above may stand for, else None."""
    if type(module) is not nn.Linear or type(x) is not torch.Tensor:  # another module may have no weight of its own
        return None
    p = module._parameters
    w, b = p.get("weight"), p.get("bias", p)   # (p: a bias that is not a parameter)
    if type(w) is not nn.Parameter or w.dim() != 2 or x.dim() != 2:
        return None
    (m, k), (n, wk) = x.shape, w.shape
    dtype, device = x.dtype, x.device
    if not (x.is_cuda and dtype in _DTYPES and w.dtype == dtype and w.device == device and device.index == torch.cuda.current_device()
            and m > 0 and k > 0 and n > 0 and wk == k and (n * x.element_size()) % 16 == 0
            and (b is None or (type(b) is nn.Parameter and b.dtype == dtype and b.device == device))
            and unhooked(module) and _ordinary_mode()):
        return None
    return w, b


def _few_for_training(m: int, narrow: int, dtype: torch.dtype) -> bool:
    """Too few rows for the passes to pay while autograd records (`narrow`: the narrower side of the Linear)."""
    if dtype == torch.float32:
        return m < LINEAR_ROWS_F32 and not any(narrow >= channels and m >= rows for channels, rows in LINEAR_ROWS_F32_WIDE)
    return m * narrow < 96 * LINEAR_ROWS_16


def linear(module: nn.Module, x: torch.Tensor, plan=None) -> torch.Tensor:
    """module(x), through the passes above where they apply; time-outs go to the plan's error word."""
    own = _own_linear(module, x)
    if own is None:
        return module(x)
    w, b = own
    if plan is None:
        plan = _plan.get()
    if not torch.is_grad_enabled() or not (x.requires_grad or w.requires_grad or (b is not None and b.requires_grad)):
        return _affine(x, w, b, plan)
    if _few_for_training(x.shape[0], min(w.shape), x.dtype) or not (b is None or b.shape == w.shape[:1]):
        return module(x)  # (the backward sums the gradient of a bias [N])
    return _Linear.apply(x, w, b, plan)


def linear_gelu(module: nn.Module, act: nn.Module, x: torch.Tensor) -> Optional[torch.Tensor]:
    """act(module(x)) in one kernel; None where that is not to be had (autograd recording, another activation, shapes)."""
    own = _own_linear(module, x) if type(act) is nn.GELU and act.approximate == "none" and unhooked(act) else None
    if own is None:
        return None
    w, b = own
    if torch.is_grad_enabled() and (x.requires_grad or w.requires_grad or (b is not None and b.requires_grad)):
        return None
    (m, k), n = x.shape, w.shape[0]
    if not _bias_ready(b, n):
        return None
    if x.dtype == torch.float32:
        # one launch for two: up to K = 256 for any number of rows (96 x 96: 1 row 6 / 6 us, 768 x 192: 16 rows 9 / 8; 96 x 384:
        # 16 rows 6 / 13)
        if not (_gemm_ready(x, w) and (k <= 256 or _gemm_pays(m, n, k))):
            return None
        fn, args = lib.ssw_gemm_f32_gelu, ()
    else:
        # N from 96 where there are many rows: a warp that drains 32 columns of a narrower tile works for less than half of them
        # (48 x 24: 60 000 rows 10 us against 14).
        # K up to 256: beyond it the library's GEMM gains more than the pass over the hidden rows costs (10 000 rows of 384:
        # 35 us against 41; of 192: 25 against 20)
        if not (k <= 256 and (n >= 96 or m <= 8192) and x.is_contiguous() and w.is_contiguous() and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0
                and n % 8 == 0 and k % 8 == 0):
            return None
        fn, args = lib.ssw_gemm_gelu, (dtype_code(x.dtype),)
    out = torch.empty((m, n), dtype=x.dtype, device=x.device)
    check(fn(ptr(x), ptr(w), ptr(b), *args, ptr(out), m, n, k, _error_word(_plan.get(), x.device), stream_ptr(x.device)), "ssw_gemm_gelu")
    return out


def layernorm_scatter(x: torch.Tensor, norm: nn.LayerNorm, parent: torch.Tensor, tap: torch.Tensor, owner: torch.Tensor) -> torch.Tensor:
    """cols [M, taps * C] with norm(x[i]) in slot (parent[i], tap[i]) and zeros elsewhere; owner [M, taps] is the
    input row of every slot (-1: none)."""
    w, b, code = norm_params(norm)
    n, c = min(x.shape[0], parent.shape[0]), x.shape[1]  # rows beyond the rulebook's voxels feed nothing
    m, taps = owner.shape
    out = torch.empty((m, taps * c), dtype=x.dtype, device=x.device)
    check(lib.ssw_layernorm_scatter(ptr(x), ptr(w), ptr(b), code, float(norm.eps), dtype_code(x.dtype), n, c, ptr(parent), ptr(tap),
                                    ptr(owner), taps, m, ptr(out), stream_ptr(x.device)), "ssw_layernorm_scatter")
    return out


def layernorm_slices(z: torch.Tensor, norm: nn.LayerNorm, parent: torch.Tensor, tap: torch.Tensor, taps: int) -> torch.Tensor:
    """out[i] = norm(z[parent[i], tap[i] * C : (tap[i] + 1) * C]), a zero row being normalised where parent[i] < 0."""
    w, b, code = norm_params(norm)
    n, c = parent.shape[0], norm.normalized_shape[0]
    out = torch.empty((n, c), dtype=z.dtype, device=z.device)
    check(lib.ssw_layernorm_slices(ptr(z), ptr(w), ptr(b), code, float(norm.eps), dtype_code(z.dtype), z.shape[0], c, ptr(parent),
                                   ptr(tap), taps, n, ptr(out), stream_ptr(z.device)), "ssw_layernorm_slices")
    return out
