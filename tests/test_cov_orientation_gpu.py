"""The covariance's orientation, C[i][j] = sum conj(x_i) x_j (not its transpose, which is the conjugate), at the sizes of
the folded triangle: small and odd T (the middle row), both kernels of the small windows, the tiles above T = 64."""

import numpy as np
import pytest
import torch

from gpu_util import call, empty, host, ptr, zeros

import holovibes_gb300 as hv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [2, 3, 7, 9, 20, 32, 33, 41, 47, 63, 64, 65, 130])
@pytest.mark.parametrize("W,H,off", [(8, 1, 0), (72, 8, 4), (200, 120, 0), (512, 504, 0), (33, 21, 0)])
def test_conjugate_of_the_first_index(cuda, T, W, H, off):
    n = W * H
    g = torch.Generator(device="cuda")
    g.manual_seed(T * 1000 + n)
    # a common component whose phase turns by 0.7 rad per frame: imaginary parts of the size of the diagonal
    base = torch.randn(n, generator=g, device="cuda", dtype=torch.complex64)
    turn = torch.polar(torch.ones(T, device="cuda"), 0.7 * torch.arange(T, device="cuda"))
    x = turn[:, None] * base + 0.3 * torch.randn(T, n, generator=g, device="cuda", dtype=torch.complex64)
    ring = torch.view_as_real(x).contiguous()
    cov = zeros(T * T * 16)
    work = empty(hv.lib().hv_pca_cov_workspace(T, n) + 16)
    # (a workspace off 16 bytes up to T = 64: the tiled kernel's planes are copied by 16-byte tensor copies)
    call("hv_pca_covariance", ring.data_ptr(), T, n, ptr(cov), ptr(work) + (off if T <= 64 else 0), None)
    got = host(cov, np.complex128, (T, T))
    z = x.to(torch.complex128)
    ref = (z.conj() @ z.T).cpu().numpy()
    # split-BF16 products lose 2^-16 of each factor's lo part (3 * 2^-16 per product at worst), the FP32
    # accumulation up to one unit per K step of 16 pixels in chains of at most 128 chunks of 4 steps
    bound = (3 * 2.0 ** -16 + 512 * 2.0 ** -23) * np.abs(np.diag(ref)).max()
    assert np.abs(got - ref).max() <= bound < 0.1 * np.abs(ref.imag).max()
