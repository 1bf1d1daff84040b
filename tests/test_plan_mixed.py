"""Plans over patterns of different kinds (host replay, no GPU): fields of a regular grid whose short
rows hold more lines than the L2, so that the batched tiles are placed field by field in bins, beside
columns stored level by level, whose tiles start again for every group of levels, on their own and together.
The fields are wrapped at fake addresses: nothing is dereferenced."""
import ctypes as C
import functools

import numpy as np
import pytest

from ghex_b200 import _capi
from ghex_b200 import unstructured as U
from ghex_b200 import workloads as W

from test_plan_check import regular_handles


def level_major_handles(doms, levels, base):
    """A float64 field per domain, vertices contiguous."""
    ctx = U.make_context(device=0)
    descs = [U.DomainDescriptor(*d) for d in doms]
    pat = U.make_pattern(ctx, U.HaloGenerator(), descs)
    keep, handles = [ctx, pat], []
    for d in descs:
        n = d.size()
        f = U.FieldDescriptor.__new__(U.FieldDescriptor)
        f.array, f._handles, f.domain_desc = None, {}, d
        f.info = {"ptr": base, "shape": (n, levels), "dtype": _capi.F64, "itemsize": 8, "device": 0}
        f.levels, f.levels_first, f.outer_stride = levels, False, 0
        base += (n * levels * 8 + 255) // 256 * 256
        keep.append(f)
        handles.append(pat(f).handle())
    return keep, handles


def checked(ctx, handles):
    n = C.c_int64()
    _capi.call("ghexb_plan_check", ctx._h, (C.c_void_p * len(handles))(*handles), len(handles), C.byref(n))
    return n.value


@pytest.mark.parametrize("levels", [1, 2, 30, 64, 65, 90, 300])
def test_level_major_tiles(levels):
    """Every halo level is checked in the forward, as an image of its owner and in the phased lists;
    the replay takes the tiles' elements as the kernels do (columns of a group of levels in turn)."""
    doms = W.config2(ni=40, nj=60, parts=4).domains
    keep, handles = level_major_handles(doms, levels, 1 << 44)
    assert checked(keep[0], handles) == 3 * levels * sum(outer.size for _, _, outer in doms)


@functools.lru_cache(maxsize=1)
def short_rows():
    """Two domains of 8 x 500 x 400 cells, halo 1 along x, periodic: 800,000 rows of one cell."""
    shape = (16, 500, 400)
    w = W.RegularWorkload("rows", shape, (True, False, False), W.regular_decomposition(shape, (2, 1, 1)))
    w.fields = [W.FieldSpec("x", np.float64, (1, 1, 0, 0, 0, 0), 1)]
    ctx, keep, handles = regular_handles(w)
    return ctx, keep, handles, checked(ctx, handles)


@pytest.mark.parametrize("levels", [65, 90, 300])
def test_binned_tiles_beside_level_major_columns(levels):
    """Short rows and a mesh in four parts, in both orders: the accesses of the plan are those of the
    two alone. (Groups of 64 levels: 65, 90 and 300 end in groups of 1, 26 and 44.)"""
    ctx, _, regular, alone = short_rows()
    keep, columns = level_major_handles(W.config2(ni=64, nj=96, parts=4).domains, levels, 1 << 44)
    alone += checked(ctx, columns)
    assert checked(ctx, regular + columns) == alone
    assert checked(ctx, columns + regular) == alone
