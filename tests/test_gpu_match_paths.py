"""Each matching path against another kernel, on references that really take it.

The box-sum kernels take dense reference lists, so the tensor-core and the
screened kernels are reached with sparse ones: fewer than one reference per 64
patch origins.  Their expected tables come from the exact warp kernel (sparse
lists of precision exact, or the patch-table entry); the number of launches
tells the paths apart.
"""

import zlib

import numpy as np
import pytest
from test_gpu_blockmatch import _patch_table, gpu_match_patches
from test_gpu_box_matching import DEV, SHAPES, SSD, _few_at_a_time, _match, _refs, _volume

pytestmark = pytest.mark.gpu


def _sparse(shape, block, rng):
    counts = [s - b + 1 for s, b in zip(shape, block)]
    lins = rng.choice(int(np.prod(counts)), size=(int(np.prod(counts)) - 1) // 64, replace=False)
    return np.stack(np.unravel_index(lins, counts), -1).astype(np.int32)


def _both(cuda, native, vol, block, radius, max_m, min_m, thr, code, refs, fast_launches, **kw):
    # (the exact warp kernel is one launch)
    from bmnd_gb300 import _abi

    runs = []
    for precision, launches in ((_abi.MATCH_EXACT, {1}), (_abi.MATCH_FAST, fast_launches)):
        before = _abi.launch_count()
        runs.append(_match(cuda, native, vol, block, radius, max_m, min_m, thr, code, precision, refs, **kw))
        assert _abi.launch_count() - before in launches
    for want, got in zip(*runs):
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("shape,block,radius", [((72, 80), (8, 8), (19, 19)), ((61, 150), (8, 8), (5, 30)),
                                                ((30, 34, 38), (5, 5, 5), (7, 7, 7)),
                                                ((32, 30, 36), (4, 4, 4), (7, 3, 5))])
@pytest.mark.parametrize("kind,max_m,frac", [("smooth", 32, 0.4), ("noise", 16, 3.0), ("offset", 32, 0.05)])
@pytest.mark.parametrize("bias", [False, True])
def test_tensor_core_ssd_of_sparse_references(cuda, native, shape, block, radius, kind, max_m, frac, bias):
    rng = np.random.default_rng(zlib.crc32(repr((shape, kind, bias)).encode()))
    vol = _volume("estimate", shape, rng)
    if kind == "noise":
        vol = rng.normal(10.0, 3.0, size=shape)
    elif kind == "offset":  # small distances under large norms
        vol = 3000.0 + 0.2 * vol
    vol = vol.astype(np.float32)
    P = int(np.prod(block))
    thr = frac * P * (float(vol.max() - vol.min()) / 8.0) ** 2
    noise = rng.uniform(0.0, 2.0, size=int(np.prod([2 * r + 1 for r in radius]))) * P if bias else None
    # norms, tile means and lists, screening, selection, exact kernel
    _both(cuda, native, vol, block, radius, max_m, 2, thr, SSD, _sparse(shape, block, rng), range(5, 20),
          noise=noise, gamma=1.5)


@pytest.mark.parametrize("shape,block,radius", [((60, 64), (8, 8), (19, 19)), ((26, 28, 30), (5, 5, 5), (7, 7, 7)),
                                                ((28, 30, 26), (4, 4, 4), (7, 7, 7)), ((20, 18, 21), (3, 4, 2), (5, 4, 6))])
@pytest.mark.parametrize("kind,max_m,min_m,thr", [("estimate", 32, 2, 0.3937), ("low", 16, 2, 0.7689),
                                                  ("counts", 16, 2, 2.9527), ("zeros", 32, 2, 0.7689),
                                                  ("estimate", 8, 4, 0.0)])
def test_screened_matching_of_sparse_references(cuda, native, shape, block, radius, kind, max_m, min_m, thr):
    rng = np.random.default_rng(zlib.crc32(repr((shape, kind, max_m)).encode()))
    vol = _volume(kind, shape, rng).astype(np.float32)
    # screening with rescoring, then the exact kernel; a count scale keeps exact requests from the tabulated terms
    _both(cuda, native, vol, block, radius, max_m, min_m, thr, DEV, _sparse(shape, block, rng), {2}, scale=1.25)


@pytest.mark.parametrize("shape,block,radius", SHAPES)
@pytest.mark.parametrize("kind,max_m,min_m,frac", [("estimate", 32, 2, 0.02), ("zeros", 32, 2, 0.4), ("low", 6, 4, 1e-7)])
@pytest.mark.parametrize("bias", [False, True])
def test_box_ssd_of_few_dense_references(cuda, native, shape, block, radius, kind, max_m, min_m, frac, bias):
    """Precision fast takes the box-sum kernels whatever the number of references;
    exact requests of so few leave them to the exact kernel."""
    from bmnd_gb300 import _abi

    rng = np.random.default_rng(zlib.crc32(repr((shape, kind, bias)).encode()))
    vol = (_volume(kind, shape, rng) - 11.0).astype(np.float32)
    refs = _refs(shape, block, rng)
    P = int(np.prod(block))
    noise = rng.uniform(0.0, 2.0, size=int(np.prod([2 * r + 1 for r in radius]))) * P if bias else None
    args = (radius, max_m, min_m, frac * P * 4.0, SSD)
    got = _match(cuda, native, vol, block, *args, _abi.MATCH_FAST, refs, noise=noise, gamma=0.7)
    want = _few_at_a_time(cuda, native, vol, block, *args, _abi.MATCH_EXACT, refs=refs, noise=noise, gamma=0.7)
    for k in (1, 2, 0):
        np.testing.assert_array_equal(got[k], want[k])


@pytest.mark.parametrize("shape,block,radius", SHAPES[:1] + SHAPES[3:5])
@pytest.mark.parametrize("kind,max_m,min_m,thr", [
    ("counts", 16, 2, 2.9527), ("bright", 16, 3, 2.9527), ("zeros", 32, 2, 0.7689), ("zeros", 7, 4, 0.0),
    ("background", 16, 2, 2.9527), ("background", 32, 4, 0.0), ("tinies", 16, 2, 2.9527), ("overflow", 16, 2, 2.0),
])
def test_log_form_equals_patch_table(cuda, native, shape, block, radius, kind, max_m, min_m, thr):
    """The screening of integer counts (precision fast takes it whatever the number
    of references), also over an empty background, whose candidates tie, and with
    values far below one among the zeros' candidates."""
    from bmnd_gb300 import _abi

    rng = np.random.default_rng(zlib.crc32(repr((shape, kind, max_m)).encode()))
    if kind in ("background", "tinies"):
        grids = np.meshgrid(*[np.linspace(-1, 1, s) for s in shape], indexing="ij")
        vol = rng.poisson(np.where(grids[0] ** 2 + grids[-1] ** 2 < 0.5, 6.0, 0.0)).astype(np.float32)
        if kind == "tinies":
            some = rng.random(shape) < 0.002
            vol[some & (vol == 0)] = rng.choice([1e-40, 1e-31, 1e-20, 1e-7, 1e-3, 0.3], size=int((some & (vol == 0)).sum()))
    else:
        vol = _volume(kind, shape, rng).astype(np.float32)
    refs = _refs(shape, block, rng)
    got = _match(cuda, native, vol, block, radius, max_m, min_m, thr, DEV, _abi.MATCH_FAST, refs)
    patches, counts = _patch_table(vol, block)
    want = gpu_match_patches(cuda, native, patches, counts, refs, radius, max_m, min_m, thr, DEV)
    for k in (1, 2, 0):
        np.testing.assert_array_equal(got[k], want[k])


@pytest.mark.parametrize("shape,block,radius,step,code,boxed", [
    ((420, 388), (8, 8), (19, 19), (3, 3), DEV, True), ((420, 388), (8, 8), (19, 19), (6, 6), DEV, False),
    ((72, 76, 70), (4, 4, 4), (7, 7, 7), (3, 3, 3), DEV, True), ((72, 76, 70), (4, 4, 4), (7, 7, 7), (3, 4, 4), DEV, False),
    ((72, 76, 70), (4, 4, 4), (7, 14, 29), (3, 3, 3), DEV, False), ((72, 76, 70), (5, 5, 5), (7, 7, 7), (3, 3, 3), SSD, True),
    ((72, 76, 70), (5, 5, 5), (1, 1, 1), (3, 3, 3), SSD, False), ((72, 76, 70), (4, 4, 4), (7, 7, 7), (4, 4, 4), SSD, True),
    ((420, 388), (8, 8), (5, 5), (3, 3), SSD, False), ((140, 140), (8, 8), (19, 19), (3, 3), SSD, False),
])
def test_exact_requests_take_the_faster_kernel(cuda, native, shape, block, radius, step, code, boxed):
    """Sparse counts, small windows and short chunks stay with the kernels of one
    reference at a time; both routes give the same tables (precision fast takes
    the box sums)."""
    from bmnd_gb300 import _abi

    rng = np.random.default_rng(zlib.crc32(repr((shape, radius, step)).encode()))
    vol = _volume("counts", shape, rng).astype(np.float32)
    axes = [np.unique(np.r_[0:s - b + 1:t, s - b]) for s, b, t in zip(shape, block, step)]
    refs = np.stack(np.meshgrid(*axes, indexing="ij"), -1).reshape(-1, len(shape)).astype(np.int32)
    args = (radius, 16, 2, 2.9527 if code == DEV else 30.0 * np.prod(block), code)
    before = _abi.launch_count()
    got = _match(cuda, native, vol, block, *args, _abi.MATCH_EXACT, refs)
    # tabulated terms: 2 launches; exact: 1; box sums: 5 and more
    assert (_abi.launch_count() - before >= 5) == boxed
    want = _match(cuda, native, vol, block, *args, _abi.MATCH_FAST, refs)
    for k in (1, 2, 0):
        np.testing.assert_array_equal(got[k], want[k])
