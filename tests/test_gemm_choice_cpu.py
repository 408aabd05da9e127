"""Which kernel a grouped GEMM of given sizes takes, checked on the CPU through the C runtime at sizes where the rows-as-N kernel and
the one-CTA kernel were timed against each other (steady loop, one B200): the slower of the two must not be the default."""
import ctypes
import os

import pytest

LIB = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "umdk_original_b200", "lib",
                   "libumdk_cam.so")


# experts, rows per expert, N, K, mode, time of the rows-as-N kernel over that of the one-CTA kernel
@pytest.mark.parametrize("e,rows,n,k,mode,ratio", [
    (256, 64, 1024, 512, 0, 2.27), (32, 100, 1024, 1024, 0, 2.00), (128, 300, 2048, 1024, 0, 1.14), (128, 100, 2048, 2048, 0, 1.14),
    (32, 100, 4096, 2048, 0, 1.06), (8, 224, 7168, 2048, 0, 1.12), (256, 64, 4096, 1024, 1, 1.16), (128, 100, 2048, 2048, 1, 1.15),
    (8, 224, 4096, 7168, 1, 1.13), (256, 8, 4096, 1536, 0, 0.86), (128, 160, 4096, 1536, 0, 0.74), (128, 32, 7168, 2048, 0, 0.77),
    (256, 160, 7168, 2048, 0, 0.77), (256, 160, 2048, 4096, 1, 0.73), (128, 128, 4096, 7168, 1, 0.73)])
def test_default_is_the_faster_form(e, rows, n, k, mode, ratio):
    if not os.path.exists(LIB):
        pytest.skip("native library not built")
    assert ctypes.CDLL(LIB).cam_grouped_gemm_rows_n_pays(e, rows, n, k, mode) == (1 if ratio < 1 else 0)
