"""The tail op at the edges of its dispatch: 16 / 28 rows per CTA, and the tensor-core kernel above one wave of the latter; the
classifier's weight gradient that it forms up to there (sums of at most 8288 products in fp32: 1e-4 of the largest element, as
every tensor of this op), and bias gradients left out."""
import numpy as np
import pytest

from zigrad_b200 import abi, opspec
from zigrad_b200.abi import SINGLE
from zigrad_b200.device import DeviceSlice

from .backends import GpuBackend
from .test_gpu_mlp_tail import H1, H2, tail_oracle
from .test_gpu_mlp_tail import test_tail_matches_the_separate_ops_of_the_oracle as check
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,ld,index", [(10, 12, False), (2, 4, True), (5, 8, "soft"), (13, 16, False)])
@pytest.mark.parametrize("side", ["16 rows", "28 rows", "last wave", "tensor cores"])
def test_rows_per_cta(gpu, side, C, ld, index):
    sms = gpu.sm_count()
    rows = {"16 rows": sms * 16 - 3, "28 rows": sms * 16 + 1, "last wave": sms * 56, "tensor cores": sms * 56 + 130}[side]
    check(gpu, rows, C, ld, index, rows, True)


def operands(be, g, rows, C, ld):
    act0 = np.maximum(g.standard_normal((rows, H1)), 0).astype(np.float32)
    W1, b1 = g.uniform(-0.2, 0.2, (H2, H1)).astype(np.float32), g.uniform(-0.1, 0.1, H2).astype(np.float32)
    W2, b2 = g.uniform(-0.3, 0.3, (C, H2)).astype(np.float32), g.uniform(-0.1, 0.1, C).astype(np.float32)
    T = np.eye(C, dtype=np.float32)[g.integers(0, C, rows)]
    ins = [be.up(x) for x in (act0, W1, b1, W2, b2, T)]
    outs = [be.up(np.zeros(s)) for s in ((rows, H2), (rows, ld), (1,), (rows, ld), (rows, H2), (rows, H1))]
    return ins, outs, tail_oracle(act0, W1, b1, W2, b2, T, rows)


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("sums", [True, False])
@pytest.mark.parametrize("side", ["one row", "16 rows", "28 rows", "last wave"])
def test_classifier_gradient(gpu, side, sums, off):
    """`off`: elements that dW2 lies past a 16-byte boundary; `sums`: with the bias gradients or without."""
    C, ld = 13, 16
    rows = {"one row": 1, "16 rows": gpu.sm_count() * 16 - 3, "28 rows": gpu.sm_count() * 16 + 1, "last wave": gpu.sm_count() * 56}[side]
    g, be = rng(rows), GpuBackend(gpu)
    assert gpu.mlp_tail_forms_dw2(rows)
    ins, outs, want = operands(be, g, rows, C, ld)
    init = g.standard_normal(off + C * H2).astype(np.float32)
    dW = be.up(init)
    dW2 = DeviceSlice(dW.ptr + 4 * off, C * H2, SINGLE, 0)
    db = [be.up(np.zeros(n)) for n in (C, H2, H1)] if sums else [None] * 3
    gpu.dispatch(opspec.mlp_tail(*ins, rows, H1, H2, C, ld, float(rows), *outs, *db, dW2=dW2))
    act1, logits, loss, dlog, dact1, dact0, db2, db1, db0 = want
    got = be.down(dW)
    np.testing.assert_array_equal(got[:off], init[:off])
    assert rel_err(got[off:].reshape(C, H2) - init[off:].reshape(C, H2), dlog.astype(np.float64).T @ act1) <= 1e-4
    assert rel_err(be.down(outs[4]).reshape(rows, H2), dact1) <= 1e-4 and rel_err(be.down(outs[5]).reshape(rows, H1), dact0) <= 1e-4
    if sums:
        for d, w in zip(db, (db2, db1, db0)):
            assert rel_err(be.down(d), w) <= 1e-4


def test_what_the_tensor_core_kernel_does_not_form(gpu):
    rows, C, ld = gpu.sm_count() * 56 + 1, 10, 12
    be = GpuBackend(gpu)
    assert not gpu.mlp_tail_forms_dw2(rows)
    ins, outs, _ = operands(be, rng(2), rows, C, ld)
    db, dW2 = [be.up(np.zeros(n)) for n in (C, H2, H1)], be.up(np.zeros(C * H2))
    for biases, grad in ((db, dW2), ([None] * 3, None), ([db[0], None, db[2]], None)):
        with pytest.raises(abi.DeviceError):
            gpu.dispatch(opspec.mlp_tail(*ins, rows, H1, H2, C, ld, float(rows), *outs, *biases, dW2=grad))
            gpu.sync()


def test_the_entry_without_a_weight_gradient_needs_every_bias_gradient(gpu):
    rows, C, ld = 64, 10, 12
    be = GpuBackend(gpu)
    ins, outs, _ = operands(be, rng(1), rows, C, ld)
    db = [be.up(np.zeros(n)) for n in (C, H2, H1)]
    for given in ([None] * 3, [db[0], db[1], None], [None, db[1], db[2]]):
        with pytest.raises(abi.DeviceError):
            gpu.L.zg_mlp_tail_fwd_bwd(SINGLE, gpu.stream, rows, H1, H2, C, *(s.ptr for s in ins), abi.LABEL_ONEHOT, ld, float(rows),
                                      *(s.ptr for s in outs), *(s.ptr if s is not None else None for s in given), 0)
            gpu.sync()
