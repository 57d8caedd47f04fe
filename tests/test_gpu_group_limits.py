"""The group filter at the ends of what a stage may ask for."""

import numpy as np
import pytest
from test_gpu_group_probe import _probe
from test_gpu_group_shapes import BLOCKS, SHAPE, _groups

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(2, 2), (16, 4), (32, 8)])
def test_covariance_table_beyond_32_bit_offsets(cuda, native, n, k):
    """A lag domain of 259^3 holds 2.17e9 coefficients of 5x5x5 patches: the rows
    of negative first-axis lags start beyond 2^31.  The same covariances over a
    domain of 29^3 (all lags of the groups are distinct in both) give the same
    noise levels, bit for bit; k = 8 takes the loop for more than four planes."""
    import bmnd_gb300 as bg
    from bmnd_gb300 import plan
    from bmnd_gb300.enums import BlockMatchDistance

    tag, big, small = "wi3d", 259, 29
    block, shape = BLOCKS[tag], SHAPE[3]
    P = int(np.prod(block))
    rng = np.random.default_rng(1000 * n + k)
    sel = _groups(rng, block, n)
    counts = tuple(s - b + 1 for s, b in zip(shape, block))
    pos = np.stack(np.unravel_index(sel, counts), -1)
    lag = pos[:, :, None] - pos[:, None]
    assert np.abs(lag).max() <= small // 2 and lag[..., 0].min() < 0
    cov = cuda.from_numpy(rng.uniform(0.5, 1.5, size=(small, small, small, P)).astype(np.float32)).cuda()
    cov[0, 0, 0] += 40.0
    wide = cuda.zeros((big, big, big, P), device="cuda")
    at = cuda.arange(-(small // 2), small // 2 + 1, device="cuda")
    for z in at:
        for y in at:
            wide[z % big, y % big, at % big] = cov[z % small, y % small, at % small]
    vol = rng.normal(50.0, 10.0, size=shape).astype(np.float32)
    full = np.full((len(sel), 32), -1, dtype=np.int32)
    full[:, :n] = sel
    res = []
    for table in (wide, cov):
        p = plan.stage_params(bg.BM4DProfile(), shape, "wiener", BlockMatchDistance.SSD, k,
                              gauss={"cov": table, "domain": tuple(table.shape[:3]), "ssd": None, "gamma": 0.0,
                                     "white_variance": None})
        res.append(_probe(cuda, p, vol, full, np.full(len(sel), n, dtype=np.int32), pilot=vol))
    np.testing.assert_array_equal(res[0]["sigma"][:, :n], res[1]["sigma"][:, :n])
    np.testing.assert_array_equal(res[0]["filt"][:, :n], res[1]["filt"][:, :n])


@pytest.mark.parametrize("block,n,k", [((8, 8, 8), 32, 2), ((8, 8, 8), 16, 5), ((6, 6, 6), 32, 8), ((7, 5, 3), 16, 9),
                                       ((6, 6), 32, 6), ((3, 2, 5), 32, 32), ((2, 2, 2), 32, 4)])
def test_exact_planes_of_other_patches_equal_the_dense_diagonal(cuda, native, block, n, k):
    """The exact variance's lists, partial sums and plane entries lie in the group
    buffers' place; the dense covariance diagonal in float64 tells whether one
    overwrites another.  With u = 2^-24 a plane's sum over a voxel's members is off
    by (n + 2) u sum |g s|, which moves the variance by at most 2 (n + 2) u sqrt(n)
    of the largest one; the sum over a warp's voxels adds U / 8 + 16 roundings."""
    import bmnd_gb300 as bg
    from bmnd_gb300 import plan, transforms
    from bmnd_gb300.enums import BlockMatchDistance
    from test_gpu_group_probe import _dense_exact_variance

    nd = len(block)
    shape = {2: (29, 33), 3: (14, 15, 17)}[nd]
    prof = (bg.BM3DProfile if nd == 2 else bg.BM4DProfile)(noise_model=bg.NoiseModel.POISSON, wiener_block_size=block)
    p = plan.stage_params(prof, shape, "wiener", BlockMatchDistance.POISSON_DEVIANCE, k)
    rng = np.random.default_rng(n + k)
    vol = rng.poisson(20.0, size=shape).astype(np.float32)
    counts = tuple(s - b + 1 for s, b in zip(shape, block))
    sel = np.full((2, p.max_stack), -1, dtype=np.int32)
    for row in sel:  # members within the search window of the first
        ref = rng.integers(0, np.array(counts))
        pos = np.clip(ref + rng.integers(-4, 5, size=(n, nd)), 0, np.array(counts) - 1)
        pos[0] = ref
        row[:n] = np.ravel_multi_index(tuple(pos.T), counts)
    sigma = _probe(cuda, p, vol, sel, np.full(2, n, dtype=np.int32), pilot=vol)["sigma"][:, :k].astype(np.float64)
    G = transforms.haar_group_matrix(n)
    spatial = [np.array(p.spatial_fwd[a][: b * b], dtype=np.float32).reshape(b, b) for a, b in enumerate(block)]
    u = 2.0 ** -24
    for group in range(2):
        pos = np.stack(np.unravel_index(sel[group, :n], counts), -1)
        dense = _dense_exact_variance(vol, block, pos, G, spatial, k).reshape(k, -1)
        np.testing.assert_allclose(sigma[group] ** 2, dense, rtol=(dense[0].size * n / 8 + 16) * u,
                                   atol=2 * (n + 2) * u * np.sqrt(n) * float(dense.max()))
