"""`dsv3_fp8_gemm_static` where the automatic plan needs more scratch than the built-in array holds: it takes fewer splits.

(tests/test_zz_no_alloc.py asks for this at K 7168, where the plan is whole tiles of 64 weight rows without any scratch.)"""
import pytest

from oracle import oracle as O
from gpu_util import assert_gemm_close
from test_zz_no_alloc import _quantised, _regular, _static

pytestmark = pytest.mark.gpu


# 72 tiles of 128 x 128 whose K (more chunks than tiles of 64 weight rows take) is split in two, 9.4 MB of partial tiles; the same number, ragged both ways
@pytest.mark.parametrize("M,N", [(384, 3072), (129, 4600)])
def test_static_scratch_gemm_takes_fewer_splits(M, N):
    from dsv3_b200 import _lib
    lib = _lib.lib
    _lib.check(lib.dsv3_set_gemm_policy(0, 0))
    K = 145 * 128
    xq, xs, wq, ws = _quantised(M, N, K, 55)
    ref, need = _regular(lib, _lib, xq, xs, wq, ws, M, N, K)
    assert need > lib.dsv3_fp8_gemm_static_scratch_bytes()
    out = _static(lib, _lib, xq, xs, wq, ws, M, N, K)
    assert_gemm_close(out, ref.cpu())
    assert_gemm_close(out, O.fp8_gemm(xq.cpu(), xs.cpu(), wq.cpu(), ws.cpu()))
