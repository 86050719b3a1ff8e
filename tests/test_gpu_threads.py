"""Two host threads, each with a context of its own, truncating spectra that
need different amounts of shared memory: neither thread's launches may depend
on what the other one's last call asked for."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_truncations_of_two_sizes_at_once():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from trim_gb300 import capi

    errors = []

    def loop(n):
        try:
            ctx = C.c_void_p()
            capi.call("tn_ctx_create", 0, C.byref(ctx))
            v = torch.linspace(1.0, 0.5, n, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            off, cnt, kept, norm = (C.c_int64 * 1)(0), (C.c_int64 * 1)(n), (C.c_int64 * 1)(), C.c_double()
            for _ in range(1500):
                capi.call("tn_truncate_sectors", ctx, 1, off, cnt, v.data_ptr(), n // 2, kept, C.byref(norm))
                assert kept[0] == n // 2
            assert abs(norm.value - 1.0) < 1e-12 and np.isfinite(v.cpu().numpy()).all()
            capi.call("tn_ctx_destroy", ctx)
        except Exception as e:  # reported by the main thread
            errors.append(repr(e))

    ts = [threading.Thread(target=loop, args=(n,)) for n in (6000, 25000)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
