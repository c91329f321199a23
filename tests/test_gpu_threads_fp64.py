"""Two handles on two host threads, FP64 calls of different sizes: the column's
shared memory depends on the batch (304 profiles x 22 channels take 32 channels
a CTA, 160 take 16), and one thread's launch must not depend on what the other
one last asked the driver for.  Outputs are the bits of the same calls alone."""
import threading

import numpy as np
import pytest

from crtmv3_gb300 import synthetic as sy

pytestmark = pytest.mark.gpu


def test_fp64_batches_of_different_sizes_on_two_threads(gpu_lib, coeff_dir):
    import torch
    import bench
    dev = torch.device("cuda")
    sensor, sizes, calls = "mwsynth_c22", (304, 160), 1500
    work = []
    for i, P in enumerate(sizes):
        atm, sfc, geo, opt = sy.clear_sky_workload(sensor, P, 100, 900 + i)
        h = gpu_lib.CRTM([sensor], coeff_dir, 0)
        b, keep, t = bench.scatter_device_inputs(torch, h, atm, sfc, geo, opt, dev)
        f64 = dict(dtype=torch.float64, device=dev)
        new = lambda: dict(radiance=torch.zeros((P, 22), **f64), bt=torch.zeros((P, 22), **f64))  # noqa: E731
        ref, out, st = new(), new(), torch.cuda.Stream()
        h.forward_device(b, ref, 0, st.cuda_stream)
        torch.cuda.synchronize()
        work.append((h, b, keep, t, ref, out, st))
    errors = []
    go = threading.Barrier(len(work))

    def loop(h, b, out, st):
        try:
            go.wait()
            for i in range(calls):
                h.forward_device(b, out, 0, st.cuda_stream)
                if i % 20 == 19:
                    st.synchronize()
        except Exception as e:   # noqa: BLE001
            errors.append(repr(e))

    threads = [threading.Thread(target=loop, args=(w[0], w[1], w[5], w[6])) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    for w in work:
        assert np.isfinite(w[4]["bt"].cpu().numpy()).all()
        for f in ("radiance", "bt"):
            assert torch.equal(w[4][f], w[5][f]), f
