"""Differentiable halo exchange for PyTorch.

    dx = DifferentiableExchange(ctx, [pattern(fd) for fd in field_descriptors])
    xs = dx(*xs)              # halo exchange in place; differentiable
    ys = stencil7(xs, 0.1)    # the 7-point update of the example program, differentiable

The forward is the exchange itself (a pure copy: every halo element takes its owner's value).
Its adjoint adds every halo gradient into the interior element it was copied from (negated where
the forward negated it, as on cubed-sphere vector components) in a fixed order — the receive
order of the pattern, the order of the CPU explicit transpose — and then zeroes the halo. It runs
in place on the incoming gradient when that has the field's layout (autograd hands each backward
a buffer of its own; a hook that retains the exchange output's gradient would see it modified).

GHEX's Python bindings have no autograd support (bindings/python/src/ghex/structured/regular.py
and unstructured.py wrap the exchange only); this module is the differentiable form of
co.exchange(pattern(field) ...).wait() on the same patterns and field descriptors.

A plan addresses fixed memory. Autograd produces new tensors at every step, so each
DifferentiableExchange keeps a small pool of plans for the forward and for the gradients, keyed by
the data pointers they are bound to (the caching allocator hands out the same few blocks step
after step); a miss rebinds the least recently used plan (ghexb_plan_rebind: a stream-ordered
rewrite of the descriptor tables). Plans hold no references to the tensors they are bound to.
"""
from __future__ import annotations

import ctypes as C
import functools
import math
import operator
from collections import OrderedDict
from typing import Any, Sequence

import torch
from torch.overrides import _get_current_function_mode_stack
from torch.utils._device import DeviceContext

from . import _capi
from ._capi import call
from ._core import BufferInfo, ExchangePlan, _flatten, _layout_of, context

__all__ = ["DifferentiableExchange", "stencil7", "Stencil7", "diffusion_program", "GraphedDiffusion"]


class _PlanPool:
    def __init__(self, ctx: context, bis: Sequence[BufferInfo], size: int):
        self.ctx, self.bis, self.size = ctx, list(bis), size
        self.plans: "OrderedDict[tuple, ExchangePlan]" = OrderedDict()
        self.hits = self.rebinds = self.created = 0

    def get(self, tensors: Sequence[torch.Tensor], stream) -> ExchangePlan:
        key = tuple(t.data_ptr() for t in tensors)
        plan = self.plans.get(key)
        if plan is not None:
            self.plans.move_to_end(key)
            self.hits += 1
            return plan
        if len(self.plans) < self.size:
            plan = ExchangePlan(self.ctx, self.bis)
            self.created += 1
        else:
            _, plan = self.plans.popitem(last=False)
        if plan.bound_pointers() != key:
            plan.rebind(tensors, stream=stream, keep=False)
            self.rebinds += 1
        self.plans[key] = plan
        return plan

    def stats(self) -> dict:
        return {"plans": len(self.plans), "hits": self.hits, "rebinds": self.rebinds, "created": self.created}


class DifferentiableExchange:
    """The halo exchange of a fixed set of buffer_infos as a differentiable function of their
    arrays. Calling it with tensors of the same layouts (shape, strides, dtype, device) as the
    fields the buffer_infos were made from exchanges those tensors in place."""

    def __init__(self, ctx: context, buffer_infos: Sequence[BufferInfo], *, graph: bool = True, pool: int = 8):
        self.context = ctx
        self._bis = _flatten(tuple(buffer_infos))
        templates = [a for bi in self._bis for a in bi.arrays()]
        for t in templates:
            if not isinstance(t, torch.Tensor):
                raise TypeError("the differentiable exchange takes torch tensors")
            if t.dtype not in (torch.float32, torch.float64):
                raise TypeError("the differentiable exchange needs float32 or float64 fields")
        self._layout = [_layout_of(t) for t in templates]
        self._tensor_layout = [(t.shape, t.stride(), t.dtype, t.device) for t in templates]
        self.graph = graph
        self._fwd = _PlanPool(ctx, self._bis, pool)
        self._bwd = _PlanPool(ctx, self._bis, pool)
        self._programs: dict = {}

    def __len__(self) -> int:
        return len(self._layout)

    def pool_stats(self) -> dict:
        """Plan-pool use of the forward exchanges and of the adjoints: lookups that found a plan
        bound to the tensors (hits) and rebinds of a plan to new memory."""
        return {"forward": self._fwd.stats(), "adjoint": self._bwd.stats()}

    def check(self, tensors: Sequence[torch.Tensor]) -> None:
        if len(tensors) != len(self._layout):
            raise ValueError(f"expected {len(self._layout)} tensors, got {len(tensors)}")
        for t, like, lay in zip(tensors, self._tensor_layout, self._layout):
            if isinstance(t, torch.Tensor) and (t.shape, t.stride(), t.dtype, t.device) == like:
                continue
            if _layout_of(t) != lay:
                raise TypeError("tensor layout differs from the field it stands for")

    def exchange_(self, tensors: Sequence[torch.Tensor]) -> None:
        """Forward exchange in place, outside autograd."""
        self.check(tensors)
        stream = torch.cuda.current_stream(tensors[0].device)
        plan = self._fwd.get(tensors, stream)
        if self.graph:
            plan.graph_launch(stream=stream)
        else:
            plan.launch(stream=stream)

    def adjoint_(self, grads: Sequence[torch.Tensor]) -> None:
        """Adjoint in place on gradient tensors of the fields' layouts, outside autograd."""
        self.check(grads)
        stream = torch.cuda.current_stream(grads[0].device)
        self._bwd.get(grads, stream).adjoint(stream=stream)

    def _finite(self, alpha: float) -> bool:
        """Whether alpha is finite in the fields' type: only then is the gradient of a halo cell that
        no interior cell lies beside zero, and the program may leave it out."""
        return math.isfinite(C.c_float(alpha).value if self._tensor_layout[0][2] == torch.float32 else alpha)

    def _program(self, halo: int):
        """The exchange and the 7-point update in fused passes, or None for an exchange that
        ghexb_program_create refuses (then the two run one after the other)."""
        if halo not in self._programs:
            program = None
            dense = all(_dense(shape, stride) for shape, stride, *_ in self._tensor_layout)
            if dense and len({dev for *_, dev in self._tensor_layout}) == 1 and self._tensor_layout[0][3].type == "cuda":
                try:
                    program = _Program(self._bis, halo)
                except _capi.GhexError as e:
                    if e.code != _capi.ERR_INVALID:
                        raise
            self._programs[halo] = program
        return self._programs[halo]

    def __call__(self, *tensors: torch.Tensor):
        if len(tensors) == 1 and isinstance(tensors[0], (list, tuple)):
            tensors = tuple(tensors[0])
        out = _ExchangeFunction.apply(self, *tensors)
        return out if isinstance(out, tuple) else (out,)


class _ExchangeFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, dx: DifferentiableExchange, *tensors):
        dx.exchange_(tensors)
        ctx.dx = dx
        ctx.mark_dirty(*tensors)
        return tensors

    @staticmethod
    def backward(ctx, *grads):
        dx: DifferentiableExchange = ctx.dx
        gs = []
        for g, (shape, stride, dtype, dev) in zip(grads, dx._tensor_layout):
            if g is not None and g.shape == shape and g.stride() == stride and g.dtype == dtype:
                gs.append(g)
                continue
            buf = torch.empty_strided(shape, stride, dtype=dtype, device=dev)
            if g is None:
                buf.zero_()
            else:
                buf.copy_(g)
            gs.append(buf)
        dx.adjoint_(gs)
        return (None, *gs)


def _launch_stencil(xs: Sequence[torch.Tensor], outs: Sequence[torch.Tensor], alpha: float, halo: int,
                    adjoint: bool) -> None:
    n = len(xs)
    if n == 0:
        return
    dtype = xs[0].dtype
    if dtype not in (torch.float32, torch.float64):
        raise TypeError("stencil7 computes in float32 or float64")
    ext, st = [], []
    for x, y in zip(xs, outs):
        if x.dim() != 3 or x.dtype != dtype or y.shape != x.shape or y.stride() != x.stride() or not x.is_cuda:
            raise TypeError("stencil7 takes 3-D CUDA tensors of one dtype")
        ext += list(x.shape)
        st += list(x.stride())
    code = _capi.F64 if dtype == torch.float64 else _capi.F32
    stream = torch.cuda.current_stream(xs[0].device).cuda_stream
    call("ghexb_stencil7", code, n, (C.c_void_p * n)(*[x.data_ptr() for x in xs]),
         (C.c_void_p * n)(*[y.data_ptr() for y in outs]), (C.c_int64 * (3 * n))(*ext), (C.c_int64 * (3 * n))(*st),
         halo, float(alpha), int(adjoint), C.c_void_p(stream))


class Stencil7(torch.autograd.Function):
    """y = x + alpha * L(x) on the interior of each domain (7-point Laplacian L), 0 on the halo."""

    @staticmethod
    def forward(ctx, alpha: float, halo: int, *xs):
        outs = [torch.empty_like(x) for x in xs]
        _launch_stencil(xs, outs, alpha, halo, adjoint=False)
        ctx.alpha, ctx.halo = alpha, halo
        ctx.layouts = [(x.shape, x.stride(), x.dtype, x.device) for x in xs]
        return tuple(outs)

    @staticmethod
    def backward(ctx, *gys):
        gin = []
        for g, (shape, stride, dtype, dev) in zip(gys, ctx.layouts):
            if g is None:
                g = torch.zeros(shape, dtype=dtype, device=dev)
            if g.stride() != stride or g.shape != shape:
                buf = torch.empty_strided(shape, stride, dtype=dtype, device=dev)
                buf.copy_(g)
                g = buf
            gin.append(g)
        outs = [torch.empty_strided(shape, stride, dtype=dtype, device=dev) for shape, stride, dtype, dev in ctx.layouts]
        _launch_stencil(gin, outs, ctx.alpha, ctx.halo, adjoint=True)
        return (None, None, *outs)


def stencil7(xs: Sequence[torch.Tensor], alpha: float = 0.1, halo: int = 1):
    out = Stencil7.apply(alpha, halo, *xs)
    return out if isinstance(out, tuple) else (out,)


@functools.lru_cache(maxsize=256)
def _dense(shape, stride) -> bool:
    """Whether torch.empty_like keeps the strides: the elements fill their memory without gaps or overlaps."""
    n = 1
    for st, size in sorted((st, size) for size, st in zip(shape, stride) if size != 1):
        if st != n:
            return False
        n *= size
    return True


class _Program:
    """The fused passes of one exchange (ghexb_program_*)."""

    def __init__(self, bis: Sequence[BufferInfo], halo: int):
        handles = (C.c_void_p * len(bis))(*[bi.handle() for bi in bis])
        h = C.c_void_p()
        call("ghexb_program_create", handles, len(bis), halo, C.byref(h))
        self._h = h
        n = C.c_int64()
        call("ghexb_program_buffer_bytes", h, C.byref(n))
        self.buffer_bytes = n.value

    def buffer(self, device) -> torch.Tensor:
        return torch.empty(self.buffer_bytes, dtype=torch.uint8, device=device)

    def steps(self, steps: int, alpha: float, stream, *, fields=None, source=None, out=None, a=None, b=None,
              adjoint: bool = False, twice: bool = False) -> None:
        def array(tensors):
            return None if tensors is None else (C.c_void_p * len(tensors))(*[t.data_ptr() for t in tensors])

        def address(t):
            return None if t is None else t.data_ptr()
        call("ghexb_program_steps", self._h, array(fields), address(source), array(out), address(a), address(b), steps,
             float(alpha), int(adjoint), int(twice), C.c_void_p(stream.cuda_stream))

    def status(self) -> int:
        """The passes' status word since it was last looked at, after a wait for the device (0: every
        load arrived in time). steps() looks at it as well, without a wait."""
        v = C.c_uint()
        call("ghexb_program_status", self._h, C.byref(v))
        return v.value

    def __del__(self, _release=_capi.release):
        _release("ghexb_program_destroy", getattr(self, "_h", None))
        self._h = None


class _Diffusion(torch.autograd.Function):
    """The program as one function: the exchange of the given tensors (their halos are the
    caller's to see), then one fused pass a step."""

    @staticmethod
    def forward(ctx, dx: DifferentiableExchange, program: _Program, steps: int, alpha: float, halo: int, *xs):
        dx.exchange_(xs)
        dev = xs[0].device
        outs = [torch.empty_like(x) for x in xs]
        a, b = (program.buffer(dev) if steps > k else None for k in (1, 2))
        program.steps(steps, alpha, torch.cuda.current_stream(dev), fields=xs, out=outs, a=a, b=b)
        ctx.dx, ctx.program, ctx.steps, ctx.alpha, ctx.halo = dx, program, steps, alpha, halo
        ctx.mark_dirty(*xs)
        ctx.set_materialize_grads(False)
        return (*xs, *outs)

    @staticmethod
    def backward(ctx, *grads):
        dx, program, steps, alpha = ctx.dx, ctx.program, ctx.steps, ctx.alpha
        n = len(dx)
        exchanged, gys = grads[:n], grads[n:]
        layouts = dx._tensor_layout
        dev = layouts[0][3]

        def like_fields(g, shape, stride, dtype, device):
            if g is not None and g.shape == shape and g.stride() == stride and g.dtype == dtype:
                return g
            buf = torch.empty_strided(shape, stride, dtype=dtype, device=device)
            return buf.zero_() if g is None else buf.copy_(g)

        def new():
            return [torch.empty_strided(shape, stride, dtype=dtype, device=device) for shape, stride, dtype, device in layouts]
        g = [like_fields(g, *lay) for g, lay in zip(gys, layouts)]
        stream = torch.cuda.current_stream(dev)
        seen = any(e is not None for e in exchanged)  # the exchanged inputs were used as well: the first step in two parts
        fused = steps - 1 if seen else steps
        if fused:
            outs = new()
            a, b = (program.buffer(dev) if fused > k else None for k in (1, 2))
            program.steps(fused, alpha, stream, fields=g, out=outs, a=a, b=b, adjoint=True)
            g = outs
        if seen:
            outs = new()
            _launch_stencil(g, outs, alpha, ctx.halo, adjoint=True)
            for o, e in zip(outs, exchanged):
                if e is not None:
                    o += e
            dx.adjoint_(outs)
            g = outs
        return (None, None, None, None, None, *g)


def diffusion_program(dx: DifferentiableExchange, xs: Sequence[torch.Tensor], steps: int = 10, alpha: float = 0.1,
                      halo: int = 1):
    """steps x (halo exchange, 7-point update); returns the final fields. The first exchange
    writes into xs: pass clones of leaf tensors that require grad. Where the exchange allows it,
    a step is one kernel (same bits). Should a kernel's load not arrive within a second, the cells
    that depend on it are not numbers, and the next program on this exchange raises GhexError."""
    xs, steps = tuple(xs), operator.index(steps)
    # (a function that changes a view in place may have one output only: a single field's exchange)
    view = torch.is_grad_enabled() and any(isinstance(x, torch.Tensor) and x.requires_grad and x._is_view() for x in xs)
    if steps > 0 and type(dx) is DifferentiableExchange and dx._finite(alpha) and not view:
        program = dx._program(halo)
        if program is not None:
            return _Diffusion.apply(dx, program, steps, alpha, halo, *xs)[len(xs):]
    for _ in range(steps):
        xs = dx(*xs)
        xs = stencil7(xs, alpha, halo)
    return xs


def _plain(xs) -> bool:
    """Ordinary CUDA tensors outside every transform and mode that sees torch's own operations
    (functorch, batched gradients, forward-mode AD, function and dispatch modes, tracing; a default
    device is no such mode: it acts on new tensors only)."""
    functorch = torch._C._functorch
    return (all(type(x) in (torch.Tensor, torch.nn.Parameter) and x.is_cuda and x.layout == torch.strided and not x.is_neg()
                and not functorch.is_functorch_wrapped_tensor(x) and not functorch.is_legacy_batchedtensor(x) for x in xs)
            and torch.autograd.forward_ad._current_level < 0 and torch._C._len_torch_dispatch_stack() == 0
            and all(type(m) is DeviceContext for m in _get_current_function_mode_stack())
            and not torch.compiler.is_compiling() and not torch.jit.is_tracing())


def _array_args(xs) -> tuple:
    n = len(xs)
    return (_capi.F64 if xs[0].dtype == torch.float64 else _capi.F32, n, (C.c_void_p * n)(*[x.data_ptr() for x in xs]),
            (C.c_int64 * (3 * n))(*[e for x in xs for e in x.shape]), (C.c_int64 * (3 * n))(*[s for x in xs for s in x.stride()]))


class _SumSquares(torch.autograd.Function):
    """The sum of squares of the interiors, and its gradient, as kernels over all domains."""

    @staticmethod
    def forward(ctx, halo: int, *xs):
        dtype, n, ptrs, ext, st = _array_args(xs)
        count = C.c_int64()
        call("ghexb_sumsq_partials", dtype, n, ext, halo, C.byref(count))
        partials = torch.empty(count.value, dtype=torch.float64, device=xs[0].device)
        out = torch.empty((), dtype=xs[0].dtype, device=xs[0].device)
        stream = torch.cuda.current_stream(xs[0].device).cuda_stream
        call("ghexb_sumsq", dtype, n, ptrs, ext, st, halo, C.c_void_p(partials.data_ptr()), count.value,
             C.c_void_p(out.data_ptr()), C.c_void_p(stream))
        ctx.save_for_backward(*xs)
        ctx.halo = halo
        return out

    @staticmethod
    def backward(ctx, g):
        xs, h = ctx.saved_tensors, ctx.halo
        # in torch's operations: a gradient that is differentiated in turn, or batched (vmap); fields
        # that a saved-tensor hook gave back as something else; and gradients of fields whose
        # strides do not suit new memory (of overlapping elements, as torch.Tensor.unfold's, two
        # gradients would share one; a slice's gradient would take the whole array's memory)
        if torch.is_grad_enabled() or not _plain((g, *xs)) or not all(
                x.dtype == g.dtype and x.device == g.device and _dense(x.shape, x.stride()) for x in xs):
            return (None, *[torch.nn.functional.pad(g * (2 * x[h:-h, h:-h, h:-h]), (h,) * 6) for x in xs])
        dtype, n, ptrs, ext, st = _array_args(xs)
        outs = [torch.empty_strided(x.shape, x.stride(), dtype=x.dtype, device=x.device) for x in xs]
        stream = torch.cuda.current_stream(xs[0].device).cuda_stream
        call("ghexb_sumsq_grad", dtype, n, ptrs, (C.c_void_p * n)(*[o.data_ptr() for o in outs]), ext, st, h,
             C.c_void_p(g.data_ptr()), C.c_void_p(stream))
        return (None, *outs)


def interior_loss(xs: Sequence[torch.Tensor], halo: int = 1) -> torch.Tensor:
    """Sum of squares of the interiors."""
    h = halo
    xs = tuple(xs)
    # (kernels are launched on the current device: tensors of another one go to torch's operations)
    if xs and h >= 1 and _plain(xs) and xs[0].get_device() == torch.cuda.current_device() and all(
            x.dim() == 3 and x.dtype in (torch.float32, torch.float64) and x.dtype == xs[0].dtype and x.device == xs[0].device
            and min(x.shape) > 2 * h and min(x.stride()) > 0 for x in xs):
        return _SumSquares.apply(h, *xs)
    return sum((x[h:-h, h:-h, h:-h] ** 2).sum() for x in xs)


class GraphedDiffusion:
    """The diffusion program (``steps`` x (halo exchange, 7-point update), loss = sum of squares of
    the final interiors) and its gradient with respect to the input fields, replayed from one CUDA
    graph on buffers of fixed memory, with the bits of ``diffusion_program``, ``interior_loss`` and
    their backward through torch.autograd.

    Where the exchange allows fused passes, a step is one kernel, forward and backward: the first
    one reads the inputs where they are (a launch of its own before the replay), the others are the
    graph's. Otherwise the graph holds the exchange and update kernels: the forward alternates two
    buffer sets; the backward seeds 2 x (final interior) and applies, for every step in reverse, the
    stencil's transpose and then the exchange's adjoint, on two more buffer sets, with four exchange
    plans of its own bound to the four sets before the capture. ``run(xs)`` returns the loss and
    the gradient (tensors the next run overwrites); a load that does not arrive is seen as by
    ``diffusion_program``."""

    def __init__(self, dx: DifferentiableExchange, templates: Sequence[torch.Tensor], steps: int = 10,
                 alpha: float = 0.1, halo: int = 1):
        templates = list(templates)
        dx.check(templates)
        steps = operator.index(steps)
        self.dx, self.steps, self.alpha, self.halo = dx, steps, alpha, halo
        dev = templates[0].device
        self._program = dx._program(halo) if steps > 0 and dx._finite(alpha) else None
        if self._program is not None:
            self._capture_fused(templates, dev)
            return

        def buffers():
            return [torch.zeros_like(t) for t in templates]
        self._inp, self._a, self._b, self._g1, self._g2 = buffers(), buffers(), buffers(), buffers(), buffers()
        stream = torch.cuda.Stream(device=dev)
        stream.wait_stream(torch.cuda.current_stream(dev))

        def plan_for(bufs):
            # a plan of its own, bound to these buffers for the graph's life (a plan of the
            # differentiable exchange's pool may be rebound to other tensors later)
            plan = ExchangePlan(dx.context, dx._bis)
            plan.rebind(bufs, stream=stream)
            return plan
        with torch.cuda.stream(stream):
            self._fwd = [plan_for(bufs) for bufs in (self._a, self._b)]
            self._bwd = [plan_for(bufs) for bufs in (self._g1, self._g2)]
            for plan in self._bwd:
                if plan.info()["adjoint_launches"] != 1:
                    raise ValueError("a graphed program needs an exchange whose adjoint is one kernel")
        torch.cuda.synchronize(dev)
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph, stream=stream):
            self.loss, self.grad = self._body()

    def _capture_fused(self, templates, dev) -> None:
        if ExchangePlan(self.dx.context, self.dx._bis).info()["adjoint_launches"] != 1:
            raise ValueError("a graphed program needs an exchange whose adjoint is one kernel")
        program, steps, alpha = self._program, self.steps, self.alpha
        self._layout = [(t.shape, t.stride(), t.dtype, t.device) for t in templates]
        self._inp = None
        self._packed = [program.buffer(dev) for _ in range(2)]
        self.grad = [torch.zeros_like(t) for t in templates]
        self.loss = torch.zeros((), dtype=templates[0].dtype, device=dev)
        dtype, n, _, ext, _ = _array_args(templates)
        count = C.c_int64()
        call("ghexb_sumsq_partials", dtype, n, ext, self.halo, C.byref(count))
        self._partials = torch.empty(count.value, dtype=torch.float64, device=dev)
        a, b = self._packed
        final = a if steps % 2 else b
        stream = torch.cuda.Stream(device=dev)
        stream.wait_stream(torch.cuda.current_stream(dev))
        torch.cuda.synchronize(dev)
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph, stream=stream):  # the first step has written a
            if steps > 1:
                program.steps(steps - 1, alpha, stream, source=a, a=a, b=b)
            call("ghexb_program_sumsq", program._h, final.data_ptr(), self._partials.data_ptr(), count.value,
                 self.loss.data_ptr(), C.c_void_p(stream.cuda_stream))
            program.steps(steps, alpha, stream, source=final, out=self.grad, a=a, b=b, adjoint=True, twice=True)

    def _body(self):
        s = torch.cuda.current_stream()
        h = self.halo
        for x, y in zip(self._a, self._inp):
            x.copy_(y)
        cur, nxt, plans = self._a, self._b, self._fwd
        for k in range(self.steps):
            plans[k % 2].launch(stream=s)
            _launch_stencil(cur, nxt, self.alpha, h, adjoint=False)
            cur, nxt = nxt, cur
        loss = interior_loss(cur, h)
        g, gn, bplans = self._g1, self._g2, self._bwd
        for gt, x in zip(g, cur):
            if self.steps > 0:
                # the last update wrote +0 on every halo cell, so doubling the whole array (exact)
                # gives the seed, 2 x on the interior and +0 elsewhere, in one kernel
                torch.mul(x, 2, out=gt)
            else:
                gt.zero_()
                gt[h:-h, h:-h, h:-h] = 2 * x[h:-h, h:-h, h:-h]
        for k in range(self.steps):
            _launch_stencil(g, gn, self.alpha, h, adjoint=True)
            bplans[(k + 1) % 2].adjoint(stream=s)
            g, gn = gn, g
        return loss, g

    def run(self, xs: Sequence[torch.Tensor]):
        if self._program is not None:
            xs = list(xs)
            if len(xs) != len(self._layout) or not all(
                    type(x) in (torch.Tensor, torch.nn.Parameter) and (x.shape, x.stride(), x.dtype, x.device) == lay
                    and not x.is_neg() for x, lay in zip(xs, self._layout)):
                if self._inp is None:  # inputs of another layout are copied into the fields' layout first
                    self._inp = [torch.zeros_like(g) for g in self.grad]
                for y, x in zip(self._inp, xs):
                    y.copy_(x)
                xs = self._inp
            self._program.steps(1, self.alpha, torch.cuda.current_stream(xs[0].device), fields=xs, a=self._packed[0])
        else:
            for y, x in zip(self._inp, xs):
                y.copy_(x)
        self.graph.replay()
        return self.loss, self.grad
