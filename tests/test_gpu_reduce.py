"""The tally reduction (GB300) at the sizes where its blocks end: one primary, around a
block of threads, around the smallest stretch of primaries per block and where the
stretches grow.  Counts are exact; each FP64 sum is compensated between threads and plain
within one (at most 256 terms, 256 x 2^-53 = 3e-14 of the magnitudes), so 1e-13 of the sum
of magnitudes is allowed against math.fsum."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 255, 256, 257, 1023, 1024, 1025, 131072, 131073, 300001])
def test_sums_at_block_edges(engine_lib, n):
    import torch
    from mytrim_gb300 import _ffi as F
    rng = np.random.default_rng(n)
    vac, coll = rng.integers(0, 5000, n), rng.integers(1, 50000, n)
    f = [rng.normal(0, 1000.0, n) for _ in range(5)]  # eel, enuc, x, y, z
    state = rng.integers(0, 5, n).astype(np.int32)
    dev = [torch.from_numpy(a).cuda() for a in (vac, coll, *f, state)]
    out = torch.full((15,), float("nan"), dtype=torch.float64, device="cuda")
    err = C.create_string_buffer(256)
    p = lambda t: C.c_void_p(t.data_ptr())
    st = F.load().mtg_reduce_primaries_noalloc(*[p(t) for t in dev], n, p(out),
                                               C.c_void_p(torch.cuda.current_stream().cuda_stream), err, len(err))
    assert st == 0, err.value
    got = out.cpu().numpy()
    rest = (state >= 1) & (state <= 3)
    want = [vac.sum(), (vac ** 2).sum(), coll.sum(), (coll ** 2).sum()]
    assert [int(v) for v in got[:4]] == [int(v) for v in want]
    assert int(got[8]) == int(rest.sum())
    cols = [f[0], f[0] ** 2, f[1], f[1] ** 2]
    for a in f[2:]:
        cols += [a[rest], a[rest] ** 2]
    for v, col in zip([*got[4:8], *got[9:]], cols):
        assert abs(v - math.fsum(col)) <= 1e-13 * math.fsum(np.abs(col))
