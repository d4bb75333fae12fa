"""Rules of the native dispatch that can be asked for without a GPU (the libraries are built and loaded, nothing is launched)."""
import ctypes

import pytest

from velox_b200.csrc import build


@pytest.fixture(scope="module")
def core():
    try:
        build.find_nvcc()
    except build.BuildError as error:
        pytest.skip(str(error))
    return build.load_core()


@pytest.mark.parametrize("N,K", [(151936, 512), (1541, 8204), (24600, 512)])
def test_rows_do_not_choose_the_float32_gemm(core, N, K):
    """A row has the same bits whatever the number of rows, so the matrix alone says which kernel it goes to; the
    scratch of the kernel on the tensor cores (none with the other) does not grow with the rows for ever."""
    ask = core.vx_gemm_f32_scratch
    ask.argtypes = [ctypes.c_void_p, ctypes.c_void_p] + [ctypes.c_int] * 4
    ask.restype = ctypes.c_longlong
    a, w = 1 << 20, 1 << 30
    pitch = (K + 7) // 8 * 8
    for rows in (17, 160, 8000, 8801, 200_000, (1 << 24) + 5, (1 << 31) - 1):
        assert ask(a, w, rows, N, K, 0) == 3 * min(rows, 8000) * pitch * 2, rows
    assert ask(a, w, 16, N, K, 0) == 0            # these are split in the kernel
    assert ask(a, w, 17, N, K, 16 * 4 + 4) == 0   # a tile of the FP32 pipes was asked for
    assert ask(a + 4, w, 17, N, K, 0) == 0 and ask(a, w + 8, 17, N, K, 0) == 0
    assert ask(a, w, 17, 512, 512, 0) == 0
