"""The product of digit operands reads its rows two entries at a time: operands
that do not allow it are not taken (no GPU)."""
import subprocess
import sys

import pytest

CALL = """
import ctypes as C
from quasix_b200 import _native
f = _native.load()._ZN2qx14gemm_nt_digitsEP6qx_ctxPKdiiS3_iiiPdi
f.restype = C.c_bool
a, lda, b, ldb = {args}
i, p = C.c_int, C.c_void_p
taken = f(p(None), p(a), i(512), i(lda), p(b), i(512), i(ldb), i(301), p(4096), i(512))
assert not taken
"""


@pytest.mark.parametrize("args", [(4096, 301, 4096, 302), (4096, 302, 4096, 301), (4104, 302, 4096, 302),
                                  (4096, 302, 4104, 302)])
def test_misaligned_rows_are_not_taken(args):
    # (In a process of its own: taken, the call would use the null context.)
    subprocess.run([sys.executable, "-c", CALL.format(args=args)], check=True)
