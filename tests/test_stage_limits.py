"""Option sets at the edge of a group's 227 KB of shared memory that a stage accepts (host side, no GPU)."""

import ctypes

import pytest

import bmnd_gb300 as bg
from bmnd_gb300 import _abi, plan
from bmnd_gb300.validation import resolve_profile


def _accepted(native, p, n_refs=1000):
    n = ctypes.c_uint64(0)
    rc = native.bmnd_stage_workspace_bytes(ctypes.byref(p), n_refs, ctypes.byref(n))
    assert rc == _abi.OK, native.bmnd_last_error()


@pytest.mark.parametrize("opts", [
    {"wiener_block_size": (8, 8, 8)},
    {"wiener_block_size": (8, 8, 8), "k": 1, "wiener_search_window": (4, 4, 4)},
    {"wiener_block_size": (8, 8, 8), "wiener_max_stack_size": 24, "k": 5, "wiener_search_window": (5, 5, 5)},
    {"wiener_block_size": (7, 7, 8), "k": 32, "wiener_search_window": (5, 5, 5)},
    {"wiener_block_size": (6, 6, 6), "k": 32, "wiener_search_window": (5, 5, 5)},
])
def test_large_patches_fit(native, opts):
    """The largest patches at stacks of 24 and 32: the exact variance's partial
    sums and plane entries must share the space of the group buffers."""
    prof = bg.BM4DProfile(noise_model="poisson", **opts)
    res = resolve_profile(prof, (64, 64, 64))
    _accepted(native, plan.stage_params(prof, (64, 64, 64), "wiener", res.blockmatch_distance, res.variance_k))


@pytest.mark.parametrize("noise,windowed,mass,k", [("poisson", 1, 1, 1), ("poisson", 0, 1, 5), ("gaussian", 1, 0, 8),
                                                   ("gaussian", 1, 1, 4)])
def test_large_patches_with_options_fit(native, noise, windowed, mass, k):
    """Windowed synthesis holds the metric diagonal, mass conservation a second
    matrix, Gaussian noise the member pairs' lags."""
    prof = bg.BM4DProfile(noise_model="poisson", wiener_block_size=(8, 8, 8), wiener_search_window=(4, 4, 4))
    res = resolve_profile(prof, (64, 64, 64))
    p = plan.stage_params(prof, (64, 64, 64), "wiener", res.blockmatch_distance, k)
    p.windowed_synthesis, p.mass_conserve = windowed, mass
    if noise == "gaussian":
        p.noise_model, p.cov_maps = _abi.NOISE_GAUSSIAN, 256
        for d in range(3):
            p.cov_domain[d] = 8
    _accepted(native, p)


def _bytes(native, prof, shape, stage, n_refs, **fields):
    res = resolve_profile(prof, shape)
    p = plan.stage_params(prof, shape, stage, res.blockmatch_distance, res.variance_k)
    for name, value in fields.items():
        setattr(p, name, value)
    n = ctypes.c_uint64(0)
    assert native.bmnd_stage_workspace_bytes(ctypes.byref(p), n_refs, ctypes.byref(n)) == _abi.OK
    return n.value


@pytest.mark.parametrize("stage", ["ht", "wiener"])
def test_tensor_core_scratch_only_where_it_is_used(native, stage):
    """A 2-D SSD stage whose matching the box-sum kernels take reserves what the
    deviance stage does; few references or a wide window keep the tensor-core
    kernels and their 4 x window bytes per reference."""
    shape, n = (2048, 2048), 900_000
    poisson = bg.BM3DProfile(noise_model="poisson", gamma=0.0)
    ssd = bg.BM3DProfile(noise_model="poisson", blockmatch_distance="ssd", gamma=0.0)
    assert _bytes(native, ssd, shape, stage, n) == _bytes(native, poisson, shape, stage, n)
    few = 2000
    assert (_bytes(native, ssd, shape, stage, few) - _bytes(native, poisson, shape, stage, few)
            >= 4 * few * 39 * 39)
    wide = bg.BM3DProfile(noise_model="poisson", blockmatch_distance="ssd", gamma=0.0,
                          **{f"{stage}_search_window": (65, 65)})
    assert _bytes(native, wide, shape, stage, n) >= 4 * n * 131 * 131


@pytest.mark.parametrize("prof,shape,n", [(bg.BM3DProfile, (512, 512), 50_000), (bg.BM4DProfile, (96, 96, 96), 60_000)])
def test_mass_conserving_stage_counts_its_matching_scratch(native, prof, shape, n):
    """Without the aggregation's region the rows of a chunk of references come from
    the workspace, not from an allocation on the stream."""
    r = (19, 19) if len(shape) == 2 else (7, 7, 7)
    extra = _bytes(native, prof(noise_model="poisson"), shape, "ht", n, mass_conserve=1)
    base = 16 * shape[0] * shape[1] * (shape[2] if len(shape) == 3 else 1)
    rows = 4 * n
    for d, v in enumerate(r):
        rows *= 2 * v + 1 if d < len(r) - 1 else (2 * v + 8) // 8 * 8
    assert extra >= base + min(rows, 1 << 28)
