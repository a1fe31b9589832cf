"""One-shot projections share a device scratch pool: concurrent calls on their own streams and
calls after the pool was returned give the serial result."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_concurrent_one_shot_projections():
    import torch

    from fastcone_b200 import _lib, ops
    from fastcone_b200.geometry import ConeGeometry

    cases = []
    for k, n in enumerate((32, 48, 64, 40)):
        ang = (np.arange(12) * (2 * np.pi / 12) + 0.1 * k).astype(np.float32)
        g = ConeGeometry((n, n, n), (3 * n // 2, n), ang, 4.0 * n, 1.0)
        vol = torch.rand(g.vol_shape, device="cuda", generator=torch.Generator("cuda").manual_seed(k))
        cases.append((g, vol, ops.project(vol, g, method=_lib.PROJ_EXPLICIT)))
    torch.cuda.synchronize()
    errors = []

    def work(k):
        try:
            g, vol, ref = cases[k]
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in range(10):
                    out = ops.project(vol, g, method=_lib.PROJ_EXPLICIT)
                    torch.cuda.current_stream().synchronize()
                    if not torch.equal(out, ref):
                        errors.append((k, i))
                    if k == 0 and i == 5:
                        _lib.lib().fcb_release_device_cache()
        except Exception as e:  # noqa: BLE001
            errors.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
