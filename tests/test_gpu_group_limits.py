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
