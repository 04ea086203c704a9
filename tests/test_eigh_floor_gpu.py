"""The floor below which the FP32 sweeps leave an entry is 5e-7 of the matrix's Frobenius norm, taken in FP64 and rounded to
a float once: 2 x 2 matrices whose off-diagonal entry is the float that the floor rounds to, or the one above it, with
the exact norm a few units of 2^-52 on that side of the rounding boundary."""

from fractions import Fraction

import numpy as np
import pytest

from gpu_util import call, dev, host, ptr, zeros

import holovibes_gb300 as hv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a,b,x", [
    ("0x1.1036fc0000000p-1", "0x1.08f2080000000p+0", "0x1.3854840000000p-21"),
    ("0x1.775fee0000000p-1", "0x1.3ba6420000000p+0", "0x1.8112be0000000p-21"),
])
def test_floor_is_an_fp64_norm(cuda, a, b, x):
    a, b, x = (float.fromhex(v) for v in (a, b, x))
    # rotated exactly if x exceeds the floor: floor = float(rel * norm) < x, i.e. rel * norm below the midpoint of x
    # and the float before it
    rel = Fraction(float(np.float32(5e-7)))
    mid = (Fraction(x) + Fraction(float(np.nextafter(np.float32(x), np.float32(0))))) / 2
    norm2 = Fraction(a) ** 2 + Fraction(b) ** 2 + 2 * Fraction(x) ** 2
    rotated = rel ** 2 * norm2 < mid ** 2
    m = np.array([[a, x], [x, b]], np.complex128)
    ev, vec, work = zeros(16), zeros(64), zeros(hv.lib().hv_pca_eigh_workspace(2))
    # no kept range: the eigenvectors are the sweeps' own
    call("hv_pca_eigh", ptr(dev(m)), 2, ptr(ev), ptr(vec), -1, -1, None, ptr(work), None)
    v = host(vec, np.complex128, (2, 2))
    assert (abs(v[0, 1]) > 0) == rotated and (abs(v[1, 0]) > 0) == rotated
