"""Which problems the small-output GEMM kernel takes (CPU: the rule is host code)."""
from ctypes import c_int

import pytest

from dhellam_b200 import kernels as K


def _ctas(M, N, Kd, out_f32=0, sms=148):
    return K.proto("dh_gemm_cluster_k", [c_int] * 5)(M, N, Kd, out_f32, sms)


@pytest.mark.parametrize("M,N,Kd,f32,want", [
    # 33 clusters of four CTAs are resident at once, 34 are not
    (128, 4096, 4096, 0, 4), (300, 1024, 1024, 0, 4), (8, 4224, 512, 0, 4), (8, 512, 8192, 1, 4), (8, 4224, 448, 0, 0),
    (64, 4352, 1024, 0, 2), (129, 2304, 512, 0, 0), (512, 1152, 1024, 0, 2), (8, 4608, 512, 1, 0), (256, 2432, 2048, 0, 2),
    (64, 8192, 12288, 0, 4), (64, 9216, 12288, 0, 2),
    # 75 to 148 tiles: the fewer rows, the longer K has to be
    (300, 6144, 4096, 0, 2), (300, 6144, 4032, 0, 0), (128, 12288, 2048, 0, 2), (128, 12288, 1984, 0, 0), (64, 16384, 2048, 0, 0),
    (24, 9600, 3072, 0, 2), (16, 12288, 3072, 0, 0), (16, 12288, 4096, 0, 2), (8, 9600, 4096, 0, 0), (8, 14336, 6144, 0, 0),
    (8, 12288, 8192, 0, 2), (8, 18816, 8192, 1, 0), (64, 12288, 4096, 1, 2),
    # more tiles than SMs, fp32 outputs of more than one row of tiles
    (300, 6528, 4096, 0, 0), (129, 1024, 4096, 1, 0)])
def test_the_rule_on_both_sides_of_its_lines(M, N, Kd, f32, want):
    assert _ctas(M, N, Kd, f32) == want
