"""Box-sum volume matching against the exact warp kernel.

Dense reference lists on the default patch shapes take the box-sum kernels
(screening by shared row sums, exact rescoring); a few references at a time on
the same volume take the exact warp kernel, one candidate after another.  The
match tables, counts and accepted counts must be equal bit for bit.
"""

import ctypes
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SSD, DEV = 0, 1


def _match(torch, native, vol, block, radius, max_m, min_m, thr, code, precision, refs, noise=None, gamma=0.0,
           scale=1.0):
    from bmnd_gb300 import _abi

    nd = vol.ndim
    counts = tuple(s - b + 1 for s, b in zip(vol.shape, block))
    p = _abi.MatchParams()
    p.ndim = nd
    for a in range(nd):
        p.counts[a], p.search_radius[a] = counts[a], radius[a]
    p.max_matches, p.min_matches, p.prefer_power_of_two = max_m, min_m, 1
    p.distance, p.stabilize_ties, p.precision, p.count_scale = code, int(code == DEV), precision, scale
    vt = torch.from_numpy(np.ascontiguousarray(vol, dtype=np.float32)).cuda()
    rt = torch.from_numpy(np.ascontiguousarray(refs, dtype=np.int32)).cuda()
    n = rt.shape[0]
    tt = torch.full((n,), float(np.float32(thr)), device="cuda")
    sel = torch.full((n, max_m), -7, dtype=torch.int32, device="cuda")
    cnt = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    acc = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    sh, bl = (ctypes.c_int32 * nd)(*vol.shape), (ctypes.c_int32 * nd)(*block)
    tail = (sel.data_ptr(), cnt.data_ptr(), acc.data_ptr(), 0)
    if noise is None:
        rc = native.bmnd_blockmatch_volume(ctypes.byref(p), vt.data_ptr(), sh, bl, rt.data_ptr(), n, tt.data_ptr(),
                                           *tail)
    else:
        nt = torch.from_numpy(np.ascontiguousarray(noise, dtype=np.float32)).cuda()
        rc = native.bmnd_blockmatch_volume_biased(ctypes.byref(p), vt.data_ptr(), sh, bl, rt.data_ptr(), n,
                                                  tt.data_ptr(), nt.data_ptr(), float(gamma), *tail)
    _abi.check(rc)
    torch.cuda.synchronize()
    return sel.cpu().numpy(), cnt.cpu().numpy(), acc.cpu().numpy()


def _few_at_a_time(torch, native, vol, block, *args, refs, **kw):
    """The exact warp kernel: fewer than one reference per 64 origins."""
    n_lins = int(np.prod([s - b + 1 for s, b in zip(vol.shape, block)]))
    step = max(1, (n_lins - 1) // 64)
    parts = [_match(torch, native, vol, block, *args, refs[i:i + step], **kw) for i in range(0, len(refs), step)]
    return tuple(np.concatenate([p[k] for p in parts]) for k in range(3))


def _volume(kind, shape, rng):
    grids = np.meshgrid(*[np.linspace(0, 1, s) for s in shape], indexing="ij")
    smooth = 5.0 + 20.0 * np.sin(3 * grids[0]) ** 2 + 10.0 * grids[-1]
    if kind == "counts":
        return rng.poisson(smooth)
    if kind == "bright":  # counts on both sides of the log form's limit
        return rng.poisson(np.where(grids[-1] > 0.5, 300.0, 1.0) * smooth)
    if kind == "estimate":
        return smooth + rng.normal(0, 0.3, size=shape)
    if kind == "low":
        return np.maximum(0.05 * smooth + rng.normal(0, 0.2, size=shape), 0.0)
    if kind == "zeros":  # exact ties, and zero patches
        return np.where(grids[-1] < 0.6, 0.0, np.rint(smooth))
    return np.where(rng.random(shape) < 0.01, 1e30, smooth)  # overflowing squares


SHAPES = [
    ((57, 203), (8, 8), (19, 19)),
    ((40, 44), (8, 8), (5, 12)),
    ((8, 131), (8, 8), (3, 19)),
    ((13, 37, 45), (5, 5, 5), (7, 7, 7)),
    ((33, 12, 40), (4, 4, 4), (7, 3, 5)),
    ((5, 70, 21), (5, 5, 5), (2, 7, 1)),
    ((70, 9, 6), (4, 4, 4), (0, 2, 7)),
]


def _refs(shape, block, rng):
    counts = [s - b + 1 for s, b in zip(shape, block)]
    lattice = np.stack(np.meshgrid(*[np.unique(np.r_[0:c:3, c - 1]) for c in counts], indexing="ij"), -1)
    lattice = lattice.reshape(-1, len(shape))
    extra = np.stack([rng.integers(0, c, size=len(lattice) // 4 + 2) for c in counts], -1)
    return np.concatenate([lattice, extra, lattice[:3]]).astype(np.int32)  # the last ones twice


@pytest.mark.parametrize("shape,block,radius", SHAPES)
@pytest.mark.parametrize("kind,max_m,min_m,thr", [
    ("counts", 16, 2, 2.9527), ("bright", 16, 2, 2.9527), ("estimate", 32, 2, 0.3937), ("estimate", 5, 3, 0.002),
    ("low", 32, 2, 0.7689), ("zeros", 32, 2, 0.7689), ("zeros", 7, 4, 0.0), ("overflow", 16, 2, 2.0),
])
def test_deviance_matching_equals_exact(cuda, native, shape, block, radius, kind, max_m, min_m, thr):
    from bmnd_gb300 import _abi

    rng = np.random.default_rng(zlib.crc32(repr((shape, kind, max_m)).encode()))
    vol = _volume(kind, shape, rng).astype(np.float32)
    refs = _refs(shape, block, rng)
    for scale in (1.0, 1.5):
        args = (radius, max_m, min_m, thr, DEV, _abi.MATCH_EXACT)
        got = _match(cuda, native, vol, block, *args, refs, scale=scale)
        want = _few_at_a_time(cuda, native, vol, block, *args, refs=refs, scale=scale)
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("shape,block,radius", SHAPES)
@pytest.mark.parametrize("kind,max_m,min_m,frac", [
    ("estimate", 32, 2, 0.02), ("estimate", 16, 2, 3.0), ("low", 6, 4, 1e-7), ("zeros", 32, 2, 0.4),
    ("overflow", 16, 2, 0.5),
])
@pytest.mark.parametrize("bias", [False, True])
def test_ssd_matching_equals_exact(cuda, native, shape, block, radius, kind, max_m, min_m, frac, bias):
    from bmnd_gb300 import _abi

    rng = np.random.default_rng(zlib.crc32(repr((shape, kind, max_m, bias)).encode()))
    vol = (_volume(kind, shape, rng) - 11.0).astype(np.float32)
    refs = _refs(shape, block, rng)
    P = int(np.prod(block))
    thr = frac * P * 4.0
    noise = rng.uniform(0.0, 2.0, size=int(np.prod([2 * r + 1 for r in radius]))) * P if bias else None
    args = (radius, max_m, min_m, thr, SSD, _abi.MATCH_EXACT)
    got = _match(cuda, native, vol, block, *args, refs, noise=noise, gamma=0.7)
    want = _few_at_a_time(cuda, native, vol, block, *args, refs=refs, noise=noise, gamma=0.7)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)


# enough references for the stages on counts, too, to take the box-sum kernels
DENSE = [
    ((57, 203), (8, 8), (19, 19)),
    ((150, 40), (8, 8), (5, 12)),
    ((13, 37, 45), (5, 5, 5), (7, 7, 7)),
    ((33, 12, 40), (4, 4, 4), (7, 3, 5)),
    ((5, 130, 70), (5, 5, 5), (2, 7, 1)),
    ((300, 9, 9), (4, 4, 4), (0, 2, 7)),
]


@pytest.mark.parametrize("shape,block,radius", DENSE)
@pytest.mark.parametrize("kind,max_m,min_m,thr", [
    ("counts", 16, 2, 2.9527), ("bright", 16, 2, 2.9527), ("estimate", 32, 2, 0.3937), ("zeros", 32, 2, 0.7689),
])
def test_dense_references_equal_exact(cuda, native, shape, block, radius, kind, max_m, min_m, thr):
    from bmnd_gb300 import _abi

    rng = np.random.default_rng(zlib.crc32(repr((shape, kind)).encode()))
    vol = _volume(kind, shape, rng).astype(np.float32)
    counts = [s - b + 1 for s, b in zip(shape, block)]
    refs = np.stack(np.meshgrid(*[np.arange(c) for c in counts], indexing="ij"), -1).reshape(-1, len(shape))
    args = (radius, max_m, min_m, thr, DEV, _abi.MATCH_EXACT)
    got = _match(cuda, native, vol, block, *args, refs)
    some = rng.choice(len(refs), size=min(len(refs), 2000), replace=False)
    want = _few_at_a_time(cuda, native, vol, block, *args, refs=refs[some])
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g[some], w)


@pytest.mark.parametrize("shape,block,radius", SHAPES)
@pytest.mark.parametrize("kind,max_m,min_m,thr", [
    ("counts", 16, 2, 2.9527), ("estimate", 32, 2, 0.3937), ("estimate", 32, 2, 0.01), ("low", 32, 2, 0.7689),
    ("flat", 32, 2, 0.7689), ("zeros", 32, 2, 0.7689), ("overflow", 16, 2, 2.0),
])
def test_real_valued_matching_equals_exact(cuda, native, shape, block, radius, kind, max_m, min_m, thr):
    """Estimates, also smooth ones that leave most of the window open."""
    from bmnd_gb300 import _abi

    rng = np.random.default_rng(zlib.crc32(repr((shape, kind, thr)).encode()))
    vol = 4.0 + rng.normal(0, 0.01, size=shape) if kind == "flat" else _volume(kind, shape, rng)
    vol = vol.astype(np.float32)
    refs = _refs(shape, block, rng)
    # a count scale other than 1: no integer-count form, whatever the values
    args = (radius, max_m, min_m, thr, DEV, _abi.MATCH_EXACT)
    got = _match(cuda, native, vol, block, *args, refs, scale=0.75)
    want = _few_at_a_time(cuda, native, vol, block, *args, refs=refs, scale=0.75)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)
