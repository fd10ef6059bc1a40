"""The SPH entry point that allocates nothing also records no profiling stages: those create events,
on the library's own device, and would end up in a caller's stream capture."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_noalloc_records_no_stage(gpulib):
    torch = pytest.importorskip("torch")
    lib = gpulib
    n, k = 1000, 7
    rng = np.random.default_rng(n)
    arrays = [rng.normal(size=(n, 3)), rng.normal(size=(n, 3)), np.ones(n),
              (np.arange(n)[:, None] + np.arange(k)[None, :]) % n, np.ones(n), np.ones(n)]
    inputs = [torch.from_numpy(a).cuda() for a in arrays]
    outputs = [torch.empty(n, m, dtype=torch.float64, device="cuda") for m in (1, 3, 1, 1)]

    def call(fn):
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert fn(n, k, *(t.data_ptr() for t in inputs), 5 / 3, 1.0, 2.0, *(t.data_ptr() for t in outputs), stream) == 0
        count = ctypes.c_int()
        out = []
        for stage in range(13):
            assert lib.gf_profile_stage(stage, None, ctypes.byref(count)) == 0
            out.append(count.value)
        return out

    lib.gf_profile(1)
    try:
        assert sum(call(lib.gf_sph_forces_noalloc_dev)) == 0
        assert sum(call(lib.gf_sph_forces_dev)) == 2  # density and force
    finally:
        lib.gf_profile(0)
