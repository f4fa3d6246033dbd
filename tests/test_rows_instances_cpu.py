"""Which instances of the products' kernels the library holds."""
import os
import subprocess

from xalm_b200 import build


def test_one_token_products_with_bf16_weights_have_an_instance_of_their_own():
    """For rows that are not whole 16-byte pieces: the instance for four tokens took 1.35 to 1.45 times as long on 14336 columns."""
    names = subprocess.run(["nm", "-C", "--defined-only", build.build_cuda()], capture_output=True, text=True, check=True).stdout
    assert "rows_matvec_kernel<__nv_bfloat16, 1, 1>" in names
    assert "rows_matvec_kernel<__nv_bfloat16, 4, 8>" in names
