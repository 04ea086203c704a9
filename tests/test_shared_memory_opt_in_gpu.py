"""Windows of very different size rendered by several threads at once: how much shared memory a kernel may take is
one attribute of the kernel on the device, so no call lowers it under another one's launch."""

import threading

import numpy as np
import pytest
import torch

from gpu_util import empty, zeros

import holovibes_gb300 as hv

pytestmark = pytest.mark.gpu


def _eigh(T):
    a = np.diag(np.arange(1.0, T + 1)).astype(np.complex128)
    cov = torch.from_numpy(a.view(np.float64)).cuda()
    ev, vec, w = zeros(T * 8), zeros(T * T * 16), zeros(T * 8)
    work = zeros(hv.lib().hv_pca_eigh_workspace(T))
    keep = (cov, ev, vec, w, work)
    return keep, lambda st: hv.lib().hv_pca_eigh(cov.data_ptr(), T, ev.data_ptr(), vec.data_ptr(), T - 1, T - 1,
                                                 w.data_ptr(), work.data_ptr(), st)


def _covariance(T):
    npix = 64
    ring, cov, work = zeros(T * npix * 8), zeros(T * T * 16), empty(hv.lib().hv_pca_cov_workspace(T, npix))
    return (ring, cov, work), lambda st: hv.lib().hv_pca_covariance(ring.data_ptr(), T, npix, cov.data_ptr(),
                                                                   work.data_ptr(), st)


def _view(T, K):
    W = H = 8
    ring, w, out = zeros(T * W * H * 8), zeros(K * T * 8), zeros(W * H * 4)
    return (ring, w, out), lambda st: hv.lib().hv_time_view(ring.data_ptr(), T, W, H, w.data_ptr(), K, hv.IMG_MODULUS, 1.0,
                                                            0, out.data_ptr(), None, st)


@pytest.mark.parametrize("large,small", [(lambda: _eigh(64), lambda: _eigh(34)), (lambda: _eigh(32), lambda: _eigh(2)),
                                         (lambda: _covariance(64), lambda: _covariance(42)),
                                         (lambda: _view(6000, 4), lambda: _view(1700, 4)),
                                         (lambda: _view(3000, 8), lambda: _view(900, 8))],
                         ids=["eigh64", "eigh32", "covariance", "view4", "view8"])
def test_threads_with_other_windows(cuda, large, small):
    calls = [large(), large(), small(), small()]
    streams = [torch.cuda.Stream() for _ in calls]
    torch.cuda.synchronize()
    status = [set() for _ in calls]

    def run(i):
        torch.cuda.set_device(0)
        for _ in range(300):
            status[i].add(calls[i][1](streams[i].cuda_stream))

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert status == [{0}] * len(calls)
