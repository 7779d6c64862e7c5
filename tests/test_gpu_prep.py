"""The layout and preparation kernels that take four points a thread, at ragged
grids (last sides of every remainder, single points, rows that allow vector loads
and rows that do not), against numpy."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [((1, 1), (16, 16)), ((5, 7), (8, 8)), ((16, 32), (16, 16)), ((33, 18), (8, 8)), ((9, 64), (16, 16)),
          ((2, 3, 5), (4, 4, 4)), ((4, 8, 12), (4, 4, 4)), ((7, 1, 9), (4, 4, 4)), ((40, 41, 44), (4, 4, 4))]


def _tiles(a, tile, pad):
    """Grid layout -> tile layout (flat), padded."""
    a = np.pad(a, [(0, -n % t) for n, t in zip(a.shape, tile)], constant_values=pad)
    nd = a.ndim
    b = a.reshape([x for n, t in zip(a.shape, tile) for x in (n // t, t)])
    return b.transpose([2 * k for k in range(nd)] + [2 * k + 1 for k in range(nd)]).reshape(-1)


def _dims(shape, tile):
    nd = len(shape)
    return nd, (ctypes.c_int * 3)(*shape, *([1] * (3 - nd))), (ctypes.c_int * 3)(*tile, *([1] * (3 - nd)))


@pytest.mark.parametrize("shape,tile", SHAPES)
def test_expand_squeeze_geom(shape, tile):
    from adaptivegriddiscretizations_b200 import _lib as L
    lib, st = L.lib(), L.stream_ptr()
    rng = np.random.default_rng(sum(shape))
    nd, cs, ct = _dims(shape, tile)
    planes = rng.standard_normal((2,) + shape).astype(np.float32)
    ref = np.stack([_tiles(p, tile, 3.5) for p in planes])
    src, dst = torch.from_numpy(planes).cuda(), torch.empty(ref.shape, device="cuda")
    L.check(lib.agd_block_expand(nd, cs, ct, 2, L.ptr(src), 0, ctypes.c_float(3.5), L.ptr(dst), st))
    assert np.array_equal(dst.cpu().numpy(), ref)
    back = torch.empty_like(src)
    L.check(lib.agd_block_squeeze(nd, cs, ct, 2, L.ptr(dst), L.ptr(back), st))
    assert np.array_equal(back.cpu().numpy(), planes)
    # an unaligned source: no vector loads
    off = torch.empty(src.numel() + 1, device="cuda")[1:]
    off.copy_(src.reshape(-1))
    L.check(lib.agd_block_expand(nd, cs, ct, 2, L.ptr(off), 0, ctypes.c_float(3.5), L.ptr(dst), st))
    assert np.array_equal(dst.cpu().numpy(), ref)
    # the dual metric of a constant and of a varying metric
    sd = nd * (nd + 1) // 2
    a = rng.standard_normal(shape + (nd, nd))
    M = np.eye(nd) + a @ np.swapaxes(a, -1, -2)
    h = np.array([0.5, 0.25, 2.0])[:nd]
    il = np.tril_indices(nd)
    m = torch.from_numpy(M[..., il[0], il[1]].astype(np.float32)).cuda().contiguous()
    dual = np.linalg.inv(M * np.outer(h, h))[..., il[0], il[1]]
    geom = torch.empty((sd, ref.shape[1]), device="cuda")
    hs = (ctypes.c_double * 3)(*h, *([1.0] * (3 - nd)))
    L.check(lib.agd_prep_geom(nd, cs, ct, L.ptr(m), 0, 0, hs, L.ptr(geom), st))
    want = np.stack([_tiles(dual[..., c], tile, np.inf) for c in range(sd)])
    got = geom.cpu().numpy()
    assert np.array_equal(np.isinf(got), np.isinf(want))
    fin = np.isfinite(want)
    # the adjugate of matrices of condition below 1e3, in float32
    assert np.abs(got[fin] - want[fin]).max() <= 1e-4 * np.abs(want[fin]).max()


@pytest.mark.parametrize("shape,tile", SHAPES)
@pytest.mark.parametrize("nseeds,cost", [(1, "field"), (3, "one"), (32, "none")])
def test_prep_args(shape, tile, nseeds, cost):
    """One launch against the separate calls, bit for bit (duplicate seeds among 32)."""
    from adaptivegriddiscretizations_b200 import _lib as L
    lib, st = L.lib(), L.stream_ptr()
    rng = np.random.default_rng(nseeds + sum(shape))
    nd, cs, ct = _dims(shape, tile)
    size = _tiles(np.zeros(shape, np.float32), tile, 0).size
    idx = np.stack([rng.integers(0, n, nseeds) for n in shape], -1).astype(np.int32)
    vals = rng.standard_normal(nseeds).astype(np.float32)
    v_t, i_t = torch.from_numpy(vals).cuda(), torch.from_numpy(idx).cuda()
    c_t = {"field": torch.rand(shape, device="cuda"), "one": torch.full((), 2.5, device="cuda"), "none": None}[cost]
    b = c_t is not None and c_t.dim() == 0
    one = torch.ones((), device="cuda")
    rhs, bits = torch.empty(size, device="cuda"), torch.empty(size // 8, dtype=torch.uint8, device="cuda")
    src = one if c_t is None else c_t
    L.check(lib.agd_block_expand(nd, cs, ct, 1, L.ptr(src), int(src.dim() == 0), ctypes.c_float(np.inf), L.ptr(rhs), st))
    L.check(lib.agd_prep_seeds(nd, cs, ct, L.ptr(i_t), L.ptr(v_t), nseeds, L.ptr(rhs), L.ptr(bits), None, st))
    for host in (False, True):
        rhs2, bits2, values = torch.empty_like(rhs), torch.empty_like(bits), torch.empty_like(rhs)
        L.check(lib.agd_prep_args(nd, cs, ct, L.ptr(c_t), int(b), idx.ctypes.data_as(ctypes.c_void_p),
                                  vals.ctypes.data_as(ctypes.c_void_p) if host else None,
                                  None if host else L.ptr(v_t), nseeds, L.ptr(values), L.ptr(rhs2), L.ptr(bits2), st))
        assert torch.equal(rhs, rhs2) and torch.equal(bits, bits2) and bool(torch.isinf(values).all())


@pytest.mark.parametrize("n", [1, 31, 2049, 1000003])
def test_nan_sum(n):
    from adaptivegriddiscretizations_b200 import _lib as L
    x = torch.rand(n, device="cuda")
    x[::7] = float("nan")
    out = torch.empty(2, dtype=torch.float64, device="cuda")
    L.check(L.lib().agd_nan_sum(L.ptr(x), n, L.ptr(out), L.stream_ptr()))
    s, c = out.tolist()
    assert c == float((~torch.isnan(x)).sum())
    assert abs(s - float(torch.nansum(x.double()))) <= 1e-12 * max(1.0, n)


@pytest.mark.parametrize("shape", [(1, 1), (9, 30), (40, 25), (5, 9, 7), (16, 20, 18)])
@pytest.mark.parametrize("npasses,cut", [(0, 0), (1, 5), (6, 30), (40, 200)])
def test_eucl_map_seeds(shape, npasses, cut):
    """The boxes around the seeds against the passes over the grid, byte for byte."""
    from adaptivegriddiscretizations_b200 import _lib as L
    lib, st = L.lib(), L.stream_ptr()
    rng = np.random.default_rng(npasses + sum(shape))
    nd, cs, _ = _dims(shape, (1,) * len(shape))
    idx = np.stack([rng.integers(0, n, 3) for n in shape], -1).astype(np.int32)
    mask = torch.zeros(shape, dtype=torch.uint8, device="cuda")
    mask[tuple(torch.from_numpy(idx.T.astype(np.int64)).cuda())] = 1
    a, b, tmp = torch.empty_like(mask), torch.empty_like(mask), torch.empty_like(mask)
    L.check(lib.agd_eucl_map(nd, cs, L.ptr(mask), npasses, cut, L.ptr(a), L.ptr(tmp), st))
    i_t = torch.from_numpy(idx).cuda()
    L.check(lib.agd_eucl_map_seeds(nd, cs, L.ptr(i_t), 3, npasses, cut, L.ptr(b), st))
    assert torch.equal(a, b)
