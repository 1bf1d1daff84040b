"""The program in fused passes (ghexb_program_*) against the exchange and the update run one after
the other, bit for bit: final fields, exchanged inputs, gradients, and the graphed loss and
gradient. The cases are where a pass can go wrong: rows that end inside a 16-byte chunk, strips and
slabs that overlap, domains two cells thick, one domain along an axis (its own neighbour), axes that
are not periodic (the halo keeps its values and its gradient), uneven domains, a halo of width 2,
more domains than one launch takes. Every value is one of the same operations with the same
roundings, so the tolerance is zero."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from ghex_b200 import _capi
from ghex_b200 import autograd as AG
from ghex_b200 import workloads as W
from ghex_b200._capi import GhexError
from ghex_b200.structured import regular as R

from gpu_helpers import RegularRun, bits_equal

pytestmark = pytest.mark.gpu

ALPHA = 0.1


def make(cuda, shape, parts, periodic, halo, dtype, seed):
    w = W.RegularWorkload("program", shape, periodic, W.regular_decomposition(shape, parts, seed))
    w.fields = [W.FieldSpec("x", dtype, (halo,) * 6, 3)]
    run = RegularRun(w, cuda)
    dx = AG.DifferentiableExchange(run.ctx, run.bis)
    gen = torch.Generator(device=cuda).manual_seed(5)
    xs = [torch.empty_like(t).uniform_(-1, 1, generator=gen) for t in run.dev["x"]]  # halos too
    return dx, xs


def separately(dx, xs, steps, halo):
    first = None
    for _ in range(steps):
        xs = dx(*xs)
        first = first or xs
        xs = AG.stencil7(xs, ALPHA, halo)
    return first, xs


def equal(a, b):
    torch.cuda.synchronize()
    return sum(bits_equal(x.detach().cpu().numpy(), y.detach().cpu().numpy()) for x, y in zip(a, b)) == 0


CASES = [
    ((16, 12, 10), (2, 2, 2), (True, True, True), 1, None),
    ((9, 11, 7), (2, 2, 2), (True, True, True), 1, None),
    ((4, 4, 4), (2, 2, 2), (True, True, True), 1, None),
    ((37, 29, 41), (3, 2, 2), (True, False, True), 1, 4),
    ((70, 33, 26), (2, 3, 1), (False, False, False), 1, 9),
    ((131, 10, 50), (1, 2, 2), (True, True, False), 1, None),
    ((24, 18, 20), (2, 2, 2), (True, False, True), 2, None),
    ((24, 20, 12), (4, 3, 3), (True, True, True), 1, None),
    ((300, 40, 9), (2, 2, 1), (True, True, True), 1, 2),
    ((270, 150, 70), (2, 1, 1), (True, True, True), 1, 3),
]


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("shape,parts,periodic,halo,seed", CASES)
def test_fused_program_bits(cuda, shape, parts, periodic, halo, seed, dtype):
    dx, x0 = make(cuda, shape, parts, periodic, halo, dtype, seed)
    assert dx._program(halo) is not None
    for steps in (1, 2, 3):
        grads, fields, ins = [], [], []
        for fused in (False, True):
            leaves = [x.clone().requires_grad_(True) for x in x0]
            xs = [x.clone() for x in leaves]
            if fused:
                ys = AG.diffusion_program(dx, xs, steps, ALPHA, halo)
                first = xs
            else:
                first, ys = separately(dx, xs, steps, halo)
            weights = [torch.linspace(-1, 1, y.numel(), dtype=y.dtype, device=cuda).reshape(y.shape) for y in ys]
            loss = sum((y * v).sum() for y, v in zip(ys, weights))
            grads.append(torch.autograd.grad(loss, leaves, retain_graph=True))
            fields.append(ys)
            ins.append(first)
            # the exchanged inputs used as well
            loss = loss + sum((x * v).sum() for x, v in zip(first, weights))
            grads[-1] += torch.autograd.grad(loss, leaves)
        assert equal(*fields)
        assert equal(*ins)
        assert equal(*grads)
    assert dx._program(halo).status() == 0


@pytest.mark.parametrize("seed", range(6))
def test_fused_program_of_other_orders(cuda, seed):
    """Two fields on uneven domains, of one pattern or two, given in any order, each in a memory order
    of its own: the images of a cell are added in the order of the exchange's adjoint."""
    rng = np.random.default_rng(seed)
    shape, parts, periodic = (31, 24, 20), (3, 2, 2), tuple(bool(v) for v in rng.integers(0, 2, 3))
    dtype = (torch.float64, torch.float32)[seed % 2]
    doms = W.regular_decomposition(shape, parts, seed)
    ctx = R.make_context()
    descs = [R.DomainDescriptor(i, (f, l)) for i, f, l in doms]
    hg = R.HaloGenerator(((0, 0, 0), tuple(n - 1 for n in shape)), (1, 1, 1), periodic)
    patterns = [R.make_pattern(ctx, hg, descs) for _ in range(2 if seed % 3 else 1)]
    gen = torch.Generator(device=cuda).manual_seed(seed)
    bound = []
    for which in range(2):
        for d, dd in zip(doms, descs):
            ext = tuple(d[2][k] - d[1][k] + 3 for k in range(3))
            order = rng.permutation(3)
            x = torch.empty([ext[k] for k in order], dtype=dtype, device=cuda).uniform_(-1, 1, generator=gen)
            x = x.permute([int(k) for k in np.argsort(order)])
            bound.append((patterns[which % len(patterns)](R.make_field_descriptor(dd, x, (1, 1, 1), ext)), x))
    if seed:
        # (fields of one pattern are paired over the domains in the order given: the first field's before the second's)
        keep = rng.permutation(len(doms))
        bound = [bound[i] for i in keep] + [bound[len(doms) + i] for i in rng.permutation(len(doms))]
    dx = AG.DifferentiableExchange(ctx, [b for b, _ in bound])
    assert dx._program(1) is not None
    check_fields_and_gradients(cuda, dx, [x for _, x in bound], 3, 1, 1)


def check_fields_and_gradients(cuda, dx, x0, steps, halo, repeats):
    leaves = [x.clone().requires_grad_(True) for x in x0]
    _, ys = separately(dx, [x.clone() for x in leaves], steps, halo)
    weights = [torch.linspace(-1, 1, y.numel(), dtype=y.dtype, device=cuda).reshape(y.shape) for y in ys]
    grads = torch.autograd.grad(sum((y * v).sum() for y, v in zip(ys, weights)), leaves)
    for _ in range(repeats):
        zs = AG.diffusion_program(dx, [x.clone() for x in leaves], steps, ALPHA, halo)
        assert equal(zs, ys)
        assert equal(torch.autograd.grad(sum((z * v).sum() for z, v in zip(zs, weights)), leaves), grads)
    assert dx._program(halo).status() == 0


@pytest.mark.parametrize("shape,parts,dtype", [
    ((48, 48, 400), (3, 3, 2), np.float64),    # 32 columns of a tile, 7 planes of a slab
    ((96, 96, 192), (3, 3, 3), np.float64),    # 64, 7
    ((64, 64, 400), (2, 2, 2), np.float64),    # 64, 6
    ((193, 79, 180), (3, 3, 2), np.float32),   # 56, 6
])
def test_tiles_of_few_columns(cuda, shape, parts, dtype):
    """Tiles that leave whole warps without a column, in slabs of more planes than are in flight: the
    cells beside a row are written by its own thread only."""
    dx, x0 = make(cuda, shape, parts, (True, True, True), 1, dtype, None)
    check_fields_and_gradients(cuda, dx, x0, 4, 1, 4)


@pytest.mark.parametrize("shape,parts,dtype", [
    ((4, 300, 8), (2, 1, 1), np.float64),      # a chunk wide, 75 strips of rows
    ((8, 300, 8), (2, 1, 1), np.float32),
    ((4, 256, 8), (1, 1, 2), np.float64),      # two chunks wide, 64 strips
    ((16, 512, 6), (2, 2, 1), np.float32),
    ((4, 252, 8), (2, 1, 1), np.float64),      # 63 strips
])
def test_narrow_long_domains(cuda, shape, parts, dtype):
    """Domains of a chunk or two along x and of more rows than a load box is high."""
    dx, x0 = make(cuda, shape, parts, (True, True, True), 1, dtype, None)
    assert dx._program(1) is not None
    check_fields_and_gradients(cuda, dx, x0, 3, 1, 1)
    graphed = AG.GraphedDiffusion(dx, x0, 3, ALPHA)
    _, ys = separately(dx, [x.clone() for x in x0], 3, 1)
    assert equal([graphed.run(x0)[0]], [AG.interior_loss(ys)])


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("shape,parts,periodic,halo,seed", CASES[:1] + CASES[3:6])
def test_graphed_program_bits(cuda, shape, parts, periodic, halo, seed, dtype):
    """Inputs of the fields' layout (read in place) and of another one (copied), and the loss
    against a sum in 64 bits: n squares added in 64 bits err by less than n roundings."""
    dx, x0 = make(cuda, shape, parts, periodic, halo, dtype, seed)
    for steps in (1, 4):
        graphed = AG.GraphedDiffusion(dx, x0, steps, ALPHA, halo)
        for scale, relaid in ((1.0, False), (-0.5, True)):
            xs = [x * scale for x in x0]
            leaves = [x.clone().requires_grad_(True) for x in xs]
            _, ys = separately(dx, [x.clone() for x in leaves], steps, halo)
            loss = AG.interior_loss(ys, halo)
            grads = torch.autograd.grad(loss, leaves)
            got, g = graphed.run([x.contiguous() for x in xs] if relaid else xs)
            assert equal([got], [loss])
            assert equal(g, grads)
            h = halo
            exact = sum((y.detach().double()[h:-h, h:-h, h:-h] ** 2).sum() for y in ys)
            n = sum(y.numel() for y in ys)
            eps = torch.finfo(loss.dtype).eps
            assert abs(loss.double() - exact) <= (n * torch.finfo(torch.float64).eps + eps) * exact


def test_interior_loss_is_differentiable_twice(cuda):
    """A gradient of the loss that is differentiated in turn: d/dx sum((dL/dx)^2) = 8 x."""
    x = torch.randn((6, 5, 7), dtype=torch.float64, device=cuda, requires_grad=True)
    (g,) = torch.autograd.grad(AG.interior_loss([x]), [x], create_graph=True)
    (gg,) = torch.autograd.grad((g ** 2).sum(), [x])
    expected = torch.zeros_like(x)
    expected[1:-1, 1:-1, 1:-1] = 8 * x.detach()[1:-1, 1:-1, 1:-1]
    assert bits_equal(gg.cpu().numpy(), expected.cpu().numpy()) == 0


@pytest.mark.parametrize("alpha", [1e39, float("inf")])
def test_alpha_beyond_the_fields_type(cuda, alpha):
    """An alpha that is infinite in single precision: the gradients of halo edges are not zero then
    (infinity times zero), and reach the cells they were copied from."""
    dx, x0 = make(cuda, (12, 10, 8), (2, 1, 1), (True, True, True), 1, np.float32, None)
    weights = [x.abs() ** 4 + 1e-3 for x in x0]  # positive, some far below their neighbours: infinite with one sign
    results = []
    for fused in (False, True):
        leaves = [x.clone().requires_grad_(True) for x in x0]
        xs = [x.clone() for x in leaves]
        if fused:
            ys = AG.diffusion_program(dx, xs, 1, alpha)
        else:
            ys = AG.stencil7(dx(*xs), alpha)
        results.append([torch.isnan(t) for t in (*ys, *torch.autograd.grad(ys, leaves, weights))])
    assert all(bool((a == b).all()) for a, b in zip(*results))
    with pytest.raises(GhexError, match="finite"):
        dx._program(1).steps(1, alpha, torch.cuda.current_stream(), fields=x0, out=[torch.empty_like(x) for x in x0])


def test_single_field_that_is_a_view(cuda):
    """One periodic domain whose field is a view in a graph: an exchange in place with one output."""
    dx, x0 = make(cuda, (9, 8, 6), (1, 1, 1), (True, True, True), 1, np.float64, None)
    assert dx._program(1) is not None
    results = []
    for program in (lambda x: AG.diffusion_program(dx, [x], 3, ALPHA), lambda x: separately(dx, [x], 3, 1)[1]):
        leaf = x0[0].clone().requires_grad_(True)
        (y,) = program(leaf.clone()[:])
        results.append([y, *torch.autograd.grad((y * y).sum(), [leaf])])
    assert equal(*results)


def test_steps_are_whole_numbers(cuda):
    """Any index counts steps; a float is refused before the inputs are touched."""
    dx, x0 = make(cuda, (12, 10, 8), (2, 1, 1), (True, True, True), 1, np.float64, None)
    xs = [x.clone() for x in x0]
    for program in (AG.diffusion_program, AG.GraphedDiffusion):
        with pytest.raises(TypeError):
            program(dx, xs, 2.0, ALPHA)
    assert equal(xs, x0)
    assert equal(AG.diffusion_program(dx, [x.clone() for x in x0], np.int64(2), ALPHA), separately(dx, xs, 2, 1)[1])


@pytest.mark.parametrize("case", ["halo", "thin", "fields of two types"])
def test_other_exchanges_run_unfused(cuda, case):
    """A pattern halo wider than the update's, domains one cell thick, fields of two types: the
    program is not fused, and is what it was."""
    if case == "halo":
        dx, xs = make(cuda, (12, 12, 12), (2, 2, 2), (True, True, True), 2, np.float64, None)
        assert dx._program(1) is None
        _, ref = separately(dx, [x.clone() for x in xs], 2, 1)
        assert equal(AG.diffusion_program(dx, [x.clone() for x in xs], 2, ALPHA, 1), ref)
    elif case == "thin":
        dx, xs = make(cuda, (8, 8, 2), (2, 2, 2), (True, True, True), 1, np.float64, None)
        assert dx._program(1) is None
        _, ref = separately(dx, [x.clone() for x in xs], 2, 1)
        assert equal(AG.diffusion_program(dx, [x.clone() for x in xs], 2, ALPHA, 1), ref)
    else:
        shape = (8, 8, 8)
        w = W.RegularWorkload("two", shape, (True,) * 3, W.regular_decomposition(shape, (2, 2, 2)))
        w.fields = [W.FieldSpec("a", np.float64, (1,) * 6, 3), W.FieldSpec("b", np.float32, (1,) * 6, 4)]
        run = RegularRun(w, cuda)
        dx = AG.DifferentiableExchange(run.ctx, run.bis)
        assert dx._program(1) is None
        with pytest.raises(TypeError, match="one dtype"):
            AG.diffusion_program(dx, run.dev["a"] + run.dev["b"], 2, ALPHA)


def loss_in_torch(xs):
    return sum((x[1:-1, 1:-1, 1:-1] ** 2).sum() for x in xs)


def same_as_torch(xs):
    """The loss and its gradients against torch's operations. The gradients are the same products;
    both sums of n squares err by less than n roundings."""
    loss, expected = AG.interior_loss(xs), loss_in_torch(xs)
    n, eps = sum(x.numel() for x in xs), torch.finfo(loss.dtype).eps
    return (abs(loss.item() - expected.item()) <= 2 * n * eps * expected.item()
            and equal(torch.autograd.grad(loss, xs), torch.autograd.grad(expected, xs)))


def test_interior_loss_of_another_device(cuda, monkeypatch):
    """Tensors that are not the current device's: torch's operations, as always."""
    xs = [torch.randn((6, 5, 7), dtype=torch.float64, device=cuda, requires_grad=True) for _ in range(2)]
    assert "SumSquares" in type(AG.interior_loss(xs).grad_fn).__name__
    assert same_as_torch(xs)
    with monkeypatch.context() as m:
        m.setattr(torch.cuda, "current_device", lambda: cuda.index + 1)
        loss = AG.interior_loss(xs)
    assert "SumSquares" not in type(loss.grad_fn).__name__
    assert equal(torch.autograd.grad(loss, xs), torch.autograd.grad(loss_in_torch(xs), xs))


def test_interior_loss_under_a_function_mode(cuda):
    """A torch function mode sees the loss's operations; a default device does not change them."""
    class Names(torch.overrides.TorchFunctionMode):
        def __init__(self):
            super().__init__()
            self.names = []

        def __torch_function__(self, func, types, args=(), kwargs=None):
            self.names.append(getattr(func, "__name__", ""))
            return func(*args, **(kwargs or {}))
    xs = [torch.randn((6, 5, 7), dtype=torch.float64, device=cuda, requires_grad=True)]
    with Names() as seen:
        loss = AG.interior_loss(xs)
    assert any("pow" in name for name in seen.names) and "sum" in seen.names
    assert equal(torch.autograd.grad(loss, xs), torch.autograd.grad(loss_in_torch(xs), xs))
    with torch.device(cuda):
        assert "SumSquares" in type(AG.interior_loss(xs).grad_fn).__name__


@pytest.mark.parametrize("strides", ["overlapping", "slice"])
def test_interior_loss_of_views(cuda, strides):
    """Fields whose elements share memory, or lie between others': every element has a gradient of its own."""
    base = torch.randn((10, 8), dtype=torch.float64, device=cuda)
    x = base.unfold(0, 4, 1) if strides == "overlapping" else torch.randn((12, 9, 14), dtype=torch.float64, device=cuda)[::2, 1:-1, ::2]
    x = x.detach().requires_grad_(True)
    assert "SumSquares" in type(AG.interior_loss([x]).grad_fn).__name__
    assert same_as_torch([x])


def test_interior_loss_with_a_batched_gradient(cuda):
    xs = [torch.randn((6, 5, 7), dtype=torch.float64, device=cuda, requires_grad=True) for _ in range(2)]
    seeds = torch.tensor([1.0, -0.5, 3.0], dtype=torch.float64, device=cuda)
    got = torch.autograd.grad(AG.interior_loss(xs), xs, seeds, is_grads_batched=True)
    assert equal(got, torch.autograd.grad(loss_in_torch(xs), xs, seeds, is_grads_batched=True))


def test_interior_loss_of_unpacked_tensors(cuda):
    """A saved-tensor hook that keeps the fields in single precision: the gradient is that of the
    fields as they were kept. One that gives them back contiguous: the gradient is the same."""
    x = torch.randn((7, 5, 6), dtype=torch.float64, device=cuda).permute(2, 1, 0).requires_grad_(True)
    for pack, kept in ((lambda t: t.float(), x.detach().float().double()), (lambda t: t.contiguous(), x.detach())):
        with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
            loss = AG.interior_loss([x])
        (g,) = torch.autograd.grad(loss, [x])
        expected = torch.zeros_like(x)
        expected[1:-1, 1:-1, 1:-1] = 2 * kept[1:-1, 1:-1, 1:-1]
        assert equal([g], [expected])


def test_a_pass_that_gave_up_is_reported(cuda):
    """The status word as a kernel leaves it when a load does not arrive, written by the host: the
    next program of the exchange raises, once, and then runs."""
    dx, x0 = make(cuda, (12, 10, 8), (2, 1, 1), (True, True, True), 1, np.float64, None)
    graphed = AG.GraphedDiffusion(dx, x0, 2, ALPHA)
    word = C.POINTER(C.c_uint)()
    _capi.call("ghexb_program_status_word", dx._program(1)._h, C.byref(word))
    _, ys = separately(dx, [x.clone() for x in x0], 2, 1)
    for program in (lambda: AG.diffusion_program(dx, [x.clone() for x in x0], 2, ALPHA), lambda: graphed.run(x0)):
        word[0] = 1
        with pytest.raises(GhexError, match="did not arrive in time"):
            program()
        program()
    assert equal(AG.diffusion_program(dx, [x.clone() for x in x0], 2, ALPHA), ys)
    word[0] = 1
    assert dx._program(1).status() == 1 and dx._program(1).status() == 0


def test_a_single_pass_out_of_place(cuda):
    """One step reads a domain's neighbours while it writes: no output may lie in any field."""
    dx, x0 = make(cuda, (12, 10, 8), (2, 1, 1), (True, True, True), 1, np.float64, None)
    program, stream = dx._program(1), torch.cuda.current_stream()
    before = [x.clone() for x in x0]
    fresh = torch.empty_like(x0[0])
    for out in (x0, [fresh, x0[0]], [x0[1], fresh]):
        with pytest.raises(GhexError, match="overlap"):
            program.steps(1, ALPHA, stream, fields=x0, out=out)
    assert equal(x0, before)
    out = [torch.empty_like(x) for x in x0]
    program.steps(1, ALPHA, stream, fields=x0, out=out)
    assert equal(out, separately(dx, before, 1, 1)[1])
