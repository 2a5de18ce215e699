"""The arrays behind an ensemble accumulator: ordinary cudaMalloc memory where a
program sees them (peer access, legacy IPC), kept for the next accumulator
where it does not, and given back.
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import alsvinn_b200 as als  # noqa: E402

pytestmark = pytest.mark.gpu

IPC_CAPABLE, MEMPOOL_HANDLE = 10, 17      # CUpointer_attribute


def _attribute(kind, ptr, ctype):
    out = ctypes.c_int(-1) if ctype is ctypes.c_int else ctype()
    fn = ctypes.CDLL("libcuda.so.1").cuPointerGetAttribute
    assert fn(ctypes.byref(out), ctypes.c_int(kind), ctypes.c_uint64(ptr)) == 0
    return out.value


@pytest.mark.parametrize("count", [1, 777, 270400, 4227136, 9000000])
def test_arrays_are_plain_device_memory(count):
    """Exportable by cudaIpcGetMemHandle, in no memory pool, each with the
    alignment of an allocation of its own, whatever the size; also after
    arrays of the size were kept."""
    for _ in range(2):
        als.MeanVariance(count).close()
        mv = als.MeanVariance(count)
        _, mean, m2 = mv.moments()
        for p in (mean, m2):
            assert p % 256 == 0
            assert _attribute(IPC_CAPABLE, p, ctypes.c_int) == 1
            assert not _attribute(MEMPOOL_HANDLE, p, ctypes.c_void_p)
        mv.close()


def test_kept_arrays_start_from_zero_and_are_given_back():
    n = 300000
    g = torch.Generator().manual_seed(1)
    a = torch.randn(70, n, generator=g, dtype=torch.float64).cuda()
    mean, var = (torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(2))
    lib = als._lib.load()
    for k in (70, 5, 64):
        mv = als.MeanVariance(n)
        mv.add(a[:k], "fp64")
        mv.result(mean, var)
        mv.close()
        x = a[:k].cpu().numpy()
        # sums of at most 70 terms: 70 x 2^-53 of values up to 6
        np.testing.assert_allclose(mean.cpu().numpy(), x.mean(0), rtol=0, atol=70 * 6 * 2.0 ** -53)
        np.testing.assert_allclose(var.cpu().numpy(), x.var(0), rtol=0, atol=4 * 70 * 36 * 2.0 ** -53)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    als.MeanVariance(4000000).close()            # 2 x 32 MB, kept
    kept = torch.cuda.mem_get_info()[0]
    als._lib.check(lib.als_scratch_trim(0, 0))
    after = torch.cuda.mem_get_info()[0]
    assert kept < after and after >= before


def test_kept_arrays_are_the_latest_and_bounded():
    """Sizes that never come back make room: after a dozen of them the arrays
    of the last accumulator are kept (a new one of its size takes no memory), at
    most 256 MiB in all."""
    lib = als._lib.load()
    torch.cuda.synchronize()
    als._lib.check(lib.als_scratch_trim(0, 0))
    start = torch.cuda.mem_get_info()[0]
    for k in range(12):
        als.MeanVariance(4000000 + 100000 * k).close()
    full = torch.cuda.mem_get_info()[0]
    assert start - full <= (256 + 16) << 20
    mv = als.MeanVariance(4000000 + 100000 * 11)
    assert torch.cuda.mem_get_info()[0] == full
    mv.close()
    als._lib.check(lib.als_scratch_trim(0, 0))
    assert torch.cuda.mem_get_info()[0] >= start - (16 << 20)


def test_seen_arrays_are_not_handed_to_the_next_accumulator():
    n = 1000003
    one = als.MeanVariance(n)
    seen = set(one.moments()[1:])
    other = als.MeanVariance(n)
    assert not seen & set(other.moments()[1:])
    one.close()
    other.close()
