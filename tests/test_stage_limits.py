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
