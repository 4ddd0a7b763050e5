"""A setup's device bytes (what the serving budget counts) against the driver's own
account of the allocation pool that its buffers come from."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu
PAGE = 2 << 20
USED_MEM_CURRENT = 7  # cudaMemPoolAttrUsedMemCurrent


def _pool_used(lib):
    assert lib.cudaDeviceSynchronize() == 0  # (frees are stream-ordered)
    pool, used = ctypes.c_void_p(), ctypes.c_uint64()
    assert lib.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert lib.cudaMemPoolGetAttribute(pool, USED_MEM_CURRENT, ctypes.byref(used)) == 0
    return used.value


@pytest.mark.parametrize("log2", [8, 11])
def test_device_bytes_are_the_pages_in_use(gpu_ctx, log2):
    import flockgpu
    lib = flockgpu.load()  # (and the CUDA runtime it links)
    before = _pool_used(lib)
    p = flockgpu.Prover(gpu_ctx, log2)
    used = _pool_used(lib) - before
    assert p.device_bytes() == -(-used // PAGE) * PAGE
    p.close()
