"""The small-window covariance (T <= 64) at the edges of its pipeline: fewer rows than converter warps, one
CTA per SM taking several parts one after another (T > 40), parts of one chunk and ragged last chunks, odd T
(the middle row of the folded triangle), a workspace off 16-byte alignment."""

import numpy as np
import pytest

from gpu_util import call, dev, empty, host, ptr, zeros

import holovibes_gb300 as hv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 3, 7, 9, 20, 32, 33, 41, 47, 63, 64])
@pytest.mark.parametrize("W,H,off", [(8, 1, 0), (72, 8, 4), (200, 120, 0), (512, 504, 0)])
def test_covariance_parts(cuda, T, W, H, off):
    import torch

    n = W * H
    g = torch.Generator(device="cuda")
    g.manual_seed(T * 1000 + n)
    ring = torch.randn(T, n, 2, generator=g, device="cuda") * 100.0
    cov = zeros(T * T * 16)
    work = empty(hv.lib().hv_pca_cov_workspace(T, n) + 16)
    call("hv_pca_covariance", ring.data_ptr(), T, n, ptr(cov), ptr(work) + off, None)
    torch.cuda.synchronize()
    got = host(cov, np.complex128, (T, T))
    x = torch.view_as_complex(ring).to(torch.complex128)
    ref = (x.conj() @ x.T).cpu().numpy()
    ref = ref if np.abs(got - ref).max() <= np.abs(got - ref.T).max() else ref.T
    assert np.array_equal(got, got.conj().T)
    # split-BF16 products lose 2^-16 of each factor's lo part (3 * 2^-16 per product relative to |a||b| at worst,
    # random signs), the FP32 accumulation up to one unit per K step of 16 pixels in chains of at most 128 chunks
    # of 4 steps: 3 * 2^-16 + 512 * 2^-23 of the diagonal
    bound = (3 * 2.0 ** -16 + 512 * 2.0 ** -23) * np.abs(np.diag(ref)).max()
    assert np.abs(got - ref).max() <= bound
