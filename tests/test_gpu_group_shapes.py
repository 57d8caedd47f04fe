"""The group filter's specialised shapes against its runtime-geometry form.

8x8, 4x4x4 and 5x5x5 patches run instantiations of their own (padded rows,
joint forward sweeps, Haar products without their zeros, exact variances from
the quarters of the Haar planes); a stage with exact risk weights runs the
runtime geometry for every shape.  Both must give the same coefficients and
noise levels.  Stationary Gaussian noise is compared with the double sum over
the covariance map in float64.
"""

import numpy as np
import pytest
from test_gpu_group_probe import _ht_margin, _params, _probe

pytestmark = pytest.mark.gpu

BLOCKS = {"ht2d": (8, 8), "ht3d": (4, 4, 4), "wi3d": (5, 5, 5)}
SHAPE = {2: (41, 47), 3: (17, 19, 23)}


def _groups(rng, block, n, count=6):
    """`count` groups of n members: a reference and members near it, some of them far apart, one of them twice."""
    shape = SHAPE[len(block)]
    counts = np.array([s - b + 1 for s, b in zip(shape, block)])
    out = []
    for k in range(count):
        ref = rng.integers(0, counts)
        reach = 2 if k % 2 else 6
        pos = np.clip(ref + rng.integers(-reach, reach + 1, size=(n, len(block))), 0, counts - 1)
        pos[0] = ref
        out.append(np.ravel_multi_index(tuple(pos.T), tuple(counts)))
    return np.array(out, dtype=np.int32)


def _run(cuda, tag, n, k, vol, sel, filt, generic):
    p = _params(tag, vol.shape, k=k, filt=filt)
    if generic:
        p.exact_risk_weights = p.weight_group_scope = p.windowed_synthesis = 1
    table = np.full((len(sel), p.max_stack), -1, dtype=np.int32)
    table[:, :n] = sel
    res = _probe(cuda, p, vol, table, np.full(len(sel), n, dtype=np.int32), pilot=vol * 0.9 + 0.5)
    return {key: v[:, :n] for key, v in res.items() if key != "weights"}


@pytest.mark.parametrize("tag", sorted(BLOCKS))
@pytest.mark.parametrize("n,k", [(1, 4), (2, 1), (2, 4), (4, 3), (8, 2), (8, 4), (16, 4), (16, 6), (16, 1), (32, 4),
                                 (32, 7), (32, 33)])
@pytest.mark.parametrize("filt", ["ht", "wiener"])
def test_specialised_shapes_equal_runtime_geometry(cuda, native, tag, n, k, filt):
    if n > _params(tag, SHAPE[len(BLOCKS[tag])]).max_stack:
        pytest.skip("beyond the profile's stack size")
    rng = np.random.default_rng(100 * n + k)
    vol = rng.poisson(20.0, size=SHAPE[len(BLOCKS[tag])]).astype(np.float32)
    sel = _groups(rng, BLOCKS[tag], n)
    got = _run(cuda, tag, n, k, vol, sel, filt, False)
    want = _run(cuda, tag, n, k, vol, sel, filt, True)
    # the same products and sums in the same order
    np.testing.assert_array_equal(got["coef"], want["coef"])
    scale = float(np.max(want["sigma"]))
    np.testing.assert_allclose(got["sigma"], want["sigma"], rtol=2e-5, atol=2e-6 * scale)
    if filt == "ht":
        decided = _ht_margin(want["coef"], want["sigma"]) > 1e-4
        assert np.array_equal(got["atten"][decided], want["atten"][decided])
    else:
        np.testing.assert_allclose(got["atten"], want["atten"], atol=1e-4)


@pytest.mark.parametrize("tag", sorted(BLOCKS))
@pytest.mark.parametrize("value", [3e30, np.inf])
def test_values_that_need_the_dense_haar_axis(cuda, native, tag, value):
    """0 x infinity and overflowing sums spread over a group as in the dense products."""
    rng = np.random.default_rng(7)
    vol = rng.poisson(20.0, size=SHAPE[len(BLOCKS[tag])]).astype(np.float32)
    vol[tuple(s // 2 for s in vol.shape)] = value
    sel = _groups(rng, BLOCKS[tag], 8, count=12)
    got = _run(cuda, tag, 8, 1, vol, sel, "ht", False)
    want = _run(cuda, tag, 8, 1, vol, sel, "ht", True)
    np.testing.assert_array_equal(got["coef"], want["coef"])


@pytest.mark.parametrize("tag", sorted(BLOCKS))
@pytest.mark.parametrize("n,k", [(1, 1), (2, 2), (2, 1), (4, 4), (4, 3), (8, 2), (8, 4), (8, 8), (8, 1)])
def test_gaussian_planes_equal_the_double_sum(cuda, native, tag, n, k):
    import bmnd_gb300 as bg
    from bmnd_gb300 import plan
    from bmnd_gb300.enums import BlockMatchDistance
    from bmnd_gb300.transforms import haar_group_matrix

    block, shape = BLOCKS[tag], SHAPE[len(BLOCKS[tag])]
    rng = np.random.default_rng(10 * n + k)
    P = int(np.prod(block))
    lag = np.stack(np.meshgrid(*[np.minimum(np.arange(s), s - np.arange(s)) for s in shape], indexing="ij"))
    cov = (np.exp(-0.4 * np.sqrt((lag ** 2).sum(0)))[..., None] * rng.uniform(0.5, 1.5, size=P)).astype(np.float32)
    table = cuda.from_numpy(cov.reshape(-1, P)).cuda()
    prof = (bg.BM3DProfile if len(block) == 2 else bg.BM4DProfile)()
    p = plan.stage_params(prof, shape, "ht" if tag.startswith("ht") else "wiener", BlockMatchDistance.SSD, k,
                          gauss={"cov": table, "domain": shape, "ssd": None, "gamma": 0.0, "white_variance": None})
    vol = rng.normal(50.0, 10.0, size=shape).astype(np.float32)
    sel = _groups(rng, block, n)
    full = np.full((len(sel), p.max_stack), -1, dtype=np.int32)
    full[:, :n] = sel
    res = _probe(cuda, p, vol, full, np.full(len(sel), n, dtype=np.int32), pilot=vol)
    G = haar_group_matrix(n).astype(np.float64)
    counts = tuple(s - b + 1 for s, b in zip(shape, block))
    kk = min(n, k)
    for group, lins in enumerate(sel):
        pos = np.stack(np.unravel_index(lins, counts), -1)
        d = (pos[:, None] - pos[None]) % np.array(shape)
        c = cov[tuple(np.moveaxis(d, -1, 0))].astype(np.float64)  # (n, n, P)
        var = np.einsum("gi,gj,ijp->gp", G[:kk], G[:kk], c)
        # n^2 terms whose magnitudes add up to at most n max C
        bound = n ** 3 * 2.0 ** -24 * float(cov.max())
        sig = res["sigma"][group, :kk].astype(np.float64)
        np.testing.assert_allclose(sig ** 2, np.maximum(var, 0.0), rtol=1e-6, atol=bound)
