"""Workspace pool of tblite_gb300_split_gemm: what it keeps, giving it back, and several threads."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


@pytest.fixture(scope="module")
def lib():
    from tblite_gb300 import _build, library

    _build.build()
    return library.load()


def _operands(torch, n, seed):
    rng = np.random.default_rng(seed)
    a, b = (torch.from_numpy(rng.standard_normal((n, n))).cuda() for _ in range(2))
    return a, b, torch.empty_like(a)


def _multiply(lib, ops, stream=None):
    a, b, c = ops
    n = a.shape[0]
    return lib.tblite_gb300_split_gemm(n, n, n, a.data_ptr(), b.data_ptr(), c.data_ptr(), 0, stream)


# one of 14 MiB of slice images, one whose 896 MiB are more than the pool may keep
@pytest.mark.parametrize("n,keeps", [(720, 512 * MIB), (5792, 512 * MIB)])
def test_memory_is_given_back(lib, n, keeps):
    import torch

    small, large = _operands(torch, 128, 1), _operands(torch, n, 2)
    assert _multiply(lib, small) == 0  # code loaded, pool made
    assert lib.tblite_gb300_split_gemm_release() == 0
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    assert _multiply(lib, large) == 0
    kept = free - torch.cuda.mem_get_info()[0]
    # (allocations are made in pieces of up to 32 MiB)
    assert kept <= keeps + 32 * MIB
    assert lib.tblite_gb300_split_gemm_release() == 0
    assert free - torch.cuda.mem_get_info()[0] <= 2 * MIB
    ref = large[1] @ large[0]
    assert _multiply(lib, large) == 0
    # slices of 56 bits: 2^-52 of the largest elements per k at most
    bound = n * 2.0 ** -52 * float(large[0].abs().max()) * float(large[1].abs().max())
    assert float((large[2] - ref).abs().max()) < bound


def test_release_while_others_multiply(lib):
    import torch

    sizes = [300, 640, 1024]
    ops = [_operands(torch, n, n) for n in sizes]
    refs = [b @ a for a, b, _ in ops]
    streams = [torch.cuda.Stream() for _ in sizes]
    torch.cuda.synchronize()
    codes = [[] for _ in sizes]

    def work(k):
        for _ in range(20):
            codes[k].append(_multiply(lib, ops[k], streams[k].cuda_stream))
            codes[k].append(lib.tblite_gb300_split_gemm_release())

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(c == 0 for cs in codes for c in cs)
    for n, (a, b, c), ref in zip(sizes, ops, refs):
        bound = n * 2.0 ** -52 * float(a.abs().max()) * float(b.abs().max())
        assert float((c - ref).abs().max()) < bound
