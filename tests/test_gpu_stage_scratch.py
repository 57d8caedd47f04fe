"""Where a stage's matching takes its scratch from: the workspace when it reaches, else the stream."""

import ctypes

import numpy as np
import pytest
from test_zz_no_alloc import _stage_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["bm3d", "bm4d"])
@pytest.mark.parametrize("stage", ["ht", "wiener"])
def test_mass_conserving_stage_matches_in_its_workspace(cuda, native, kind, stage):
    """No allocation with the workspace the library asks for; the same match tables
    with a smaller one, whose missing part it allocates."""
    import bmnd_gb300 as bg
    from bmnd_gb300 import _abi

    shape, prof = ((200, 180), bg.BM3DProfile) if kind == "bm3d" else ((56, 62, 70), bg.BM4DProfile)
    rng = np.random.default_rng(len(shape))
    noisy = rng.poisson(10.0 + 5.0 * np.linspace(0, 1, shape[0]).reshape((-1,) + (1,) * (len(shape) - 1)),
                        size=shape).astype(np.float32)
    p, refs_h = _stage_inputs(stage, noisy, prof(noise_model="poisson"))
    p.mass_conserve = 1
    x = cuda.from_numpy(noisy).cuda()
    refs, n = cuda.from_numpy(refs_h).cuda(), refs_h.shape[0]
    need = ctypes.c_uint64(0)
    _abi.check(native.bmnd_stage_workspace_bytes(ctypes.byref(p), n, ctypes.byref(need)))
    tables, allocs = [], []
    # the float64 accumulators, the match table and small tables, then the full workspace
    least = 16 * noisy.size + 4 * n * (p.max_stack + 2) + (1 << 20)
    assert least < need.value
    for size in (need.value, least):
        ws = cuda.empty(size, dtype=cuda.uint8, device="cuda")
        out = cuda.empty_like(x)
        sel = cuda.full((n, p.max_stack), -7, dtype=cuda.int32, device="cuda")
        cnt = cuda.full((n,), -7, dtype=cuda.int32, device="cuda")
        before = _abi.device_alloc_count()
        _abi.check(native.bmnd_stage(ctypes.byref(p), x.data_ptr(), x.data_ptr(), refs.data_ptr(), n, out.data_ptr(),
                                     sel.data_ptr(), cnt.data_ptr(), None, ws.data_ptr(), size, 0))
        cuda.cuda.synchronize()
        allocs.append(_abi.device_alloc_count() - before)
        tables.append((sel.cpu().numpy(), cnt.cpu().numpy()))
    assert allocs == [0, 1]
    np.testing.assert_array_equal(tables[0][1], tables[1][1])
    np.testing.assert_array_equal(tables[0][0], tables[1][0])
