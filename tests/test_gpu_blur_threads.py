"""Blurs of different kernel sizes from several host threads at once: each one's result is that of the call alone."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("separable", [True, False])
def test_blurs_from_several_threads(separable):
    from cardiax_gb300 import _native as N
    from cardiax_gb300.tissue import stream_handle
    H, W, calls = 70, 66, 1500
    g = torch.Generator().manual_seed(3)
    plane = torch.rand((H, W), generator=g).cuda()
    sizes = (9, 510, 33, 300) if separable else (9, 200, 33, 120)
    jobs = []
    for K in sizes:
        w = torch.rand((2, K) if separable else (K, K), generator=g).cuda()
        jobs.append((K, w, torch.empty_like(plane), torch.empty_like(plane)))

    def call(K, w, tmp, out, stream):
        if separable:
            return N.lib().fk_conv2d_separable(plane.data_ptr(), H, W, W, w[0].data_ptr(), w[1].data_ptr(), K,
                                               tmp.data_ptr(), W, out.data_ptr(), W, 0, stream)
        return N.lib().fk_conv2d_same(plane.data_ptr(), H, W, W, w.data_ptr(), K, out.data_ptr(), W, 0, stream)

    want = []
    for job in jobs:
        assert call(*job, stream_handle()) == 0
        want.append(job[3].clone())
    torch.cuda.synchronize()
    failed = []

    def work(job):
        s = torch.cuda.Stream()
        for k in range(calls):
            rc = call(*job, s.cuda_stream)
            if rc:
                failed.append((job[0], rc))
                break
            if k % 100 == 99:
                s.synchronize()
        s.synchronize()

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for job, ref in zip(jobs, want):
        assert torch.equal(job[3], ref)
