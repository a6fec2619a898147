"""Split products of long rows whose digits all have one sign: the largest sums there are (needs a GPU).

Constant rows and columns, up to the longest accepted inner dimension.  The exact levels hold their
sums as integers.  The last two levels add up in FP32 over all of k: at most 7 products of digits below
2^7 per k in either, so sums below 2^(17 + log2 k), to which each of the 7 k / 16 instructions adds with
an error of one unit in the last place at most; the levels stand 2^-40 and 2^-48 below the leading one,
whose unit is 2^-14 of the scale.  The dropped products are below 2^-51 of the scale per k.  Elements
lie between half the scale and the scale, so both are taken against four times |a| |b|.
"""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [385, 3072, 12287, 12288])
@pytest.mark.parametrize("sym", [False, True])
def test_constant_rows(k, sym):
    import torch

    from tblite_gb300 import library

    lib = library.load()
    rng = np.random.default_rng(k)
    m, n = (130, 130) if sym else (130, 66)
    a = rng.uniform(0.5, 1.0, m)
    a[0], a[1] = np.nextafter(1.0, 0.0), 0.5
    b = a if sym else rng.uniform(0.5, 1.0, n)
    ta = torch.from_numpy(a).cuda().expand(k, m).contiguous()  # column-major m x k
    tb = torch.from_numpy(b).cuda()[:, None].expand(n, k).contiguous()  # column-major k x n
    tc = torch.full((n, m), np.nan, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert lib.tblite_gb300_split_gemm(m, n, k, ctypes.c_void_p(ta.data_ptr()),
                                       ctypes.c_void_p(tb.data_ptr()),
                                       ctypes.c_void_p(tc.data_ptr()), int(sym), None) == 0
    c = tc.cpu().numpy().T.astype(np.longdouble)
    ref = np.longdouble(k) * np.outer(a.astype(np.longdouble), b.astype(np.longdouble))
    ulp = 2.0 ** (math.ceil(17 + math.log2(k)) - 24)
    low = 7 * k / 16 * ulp * (2.0 ** -54 + 2.0 ** -62)
    bound = 4.0 * (low / k + 2.0 ** -51) + 2.0 ** -53
    assert float(np.max(np.abs(c - ref) / ref)) <= bound
