"""SpMV at both sides of the rule on the rows per SM (148 x 512 rows) for every block width with its
own kernel, with rows of one to nine blocks."""
import ctypes

import numpy as np
import pytest

from bosss_b200 import _capi as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [35 * 20, 148 * 512 + 35])
@pytest.mark.parametrize("bc", [4, 10, 20, 35])
def test_spmv_rows(bc, rows):
    br = bc
    nb = -(-rows // br)
    r = np.random.default_rng(bc)
    # hex-like rows of nine blocks, a few with fewer (padding stays below a quarter)
    cnt = np.where(r.uniform(size=nb) < 0.1, r.integers(1, 9, nb), 9)
    rp = np.zeros(nb + 1, np.int64)
    rp[1:] = np.cumsum(cnt)
    ci = r.integers(0, nb, rp[-1]).astype(np.int32)
    v = r.uniform(-1, 1, (rp[-1], br, bc))
    x, y0 = r.uniform(-1, 1, nb * bc), r.uniform(-1, 1, nb * br)
    prod = np.einsum("nij,nj->ni", v, x.reshape(nb, bc)[ci])
    ref = np.zeros((nb, br))
    np.add.at(ref, np.repeat(np.arange(nb), cnt), prod)
    A = ctypes.c_void_p()
    C.check(C.lib().bosss_b200_bsr_create(nb, nb, br, bc, C.ptr(rp), C.ptr(ci), C.ptr(v), 0, ctypes.byref(A)))
    try:
        y = y0.copy()
        C.check(C.lib().bosss_b200_bsr_spmv(A, 0.5, C.ptr(x), -2.0, C.ptr(y)))
    finally:
        C.lib().bosss_b200_bsr_destroy(A)
    want = 0.5 * ref.ravel() - 2.0 * y0
    # 9 bc products of size <= 1 per row: rounding below (9 bc) 2^-53, relative to a norm of order one
    assert np.linalg.norm(y - want) <= 1e-14 * np.linalg.norm(want)
