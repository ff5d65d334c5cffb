"""The tail op at the edges of its dispatch: 16 / 28 rows per CTA, and the tensor-core kernel above one wave of the latter."""
import pytest

from .test_gpu_mlp_tail import test_tail_matches_the_separate_ops_of_the_oracle as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,ld,index", [(10, 12, False), (2, 4, True), (5, 8, "soft"), (13, 16, False)])
@pytest.mark.parametrize("side", ["16 rows", "28 rows", "last wave", "tensor cores"])
def test_rows_per_cta(gpu, side, C, ld, index):
    sms = gpu.sm_count()
    rows = {"16 rows": sms * 16 - 3, "28 rows": sms * 16 + 1, "last wave": sms * 56, "tensor cores": sms * 56 + 130}[side]
    check(gpu, rows, C, ld, index, rows, True)
