"""The cross filter's decode of a normal code on the GPU: the quotient by 32767 for
every 16-bit half against the IEEE division, and the normals against the
reference's expressions in NumPy."""
import numpy as np
import pytest
import torch

from sensemap_b200 import _native as N

pytestmark = pytest.mark.gpu


def test_every_half_of_a_code_is_divided_exactly():
    half = np.arange(65536, dtype=np.uint32)
    other = np.random.default_rng(0).permutation(half)
    codes = torch.from_numpy(((half << 16) | other).view(np.int32)).cuda()
    quotients = torch.empty(2 * len(half), device="cuda")
    normals = torch.empty(3 * len(half), device="cuda")
    N.check(N.lib().smvs_test_decode_codes(codes.data_ptr(), len(half), quotients.data_ptr(), normals.data_ptr(), None))
    q = quotients.cpu().numpy().reshape(-1, 2)
    for got, iq in zip(q.T, (half, other)):
        want = iq.astype(np.float32) / np.float32(32767)
        np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
    # kernel_functions.cu:3592-3601; the sum of squares is fused there as here.
    q1, q2 = (q - np.float32(1)).T
    s = (q1.astype(np.float64) * q1 + (q2 * q2).astype(np.float64)).astype(np.float32)
    ok = s <= 1
    z = (1.0 - 2.0 * s.astype(np.float64)).astype(np.float32)
    n = normals.cpu().numpy().reshape(-1, 3)
    assert ok.sum() > 30000
    np.testing.assert_array_equal(n[ok, 0], z[ok])
    assert np.isnan(n[s > 1, 1]).all()
