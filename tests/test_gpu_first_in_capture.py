"""Ops whose first call on a stream happens inside a capture, where no work space can be grown: those that need none of
their own, or that find enough of it, are captured."""
import numpy as np
import pytest

from zigrad_b200 import opspec
from zigrad_b200.device import CudaDevice

from .backends import OracleBackend
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


@pytest.fixture()
def fresh(gpu):
    """A device whose stream has not been used before."""
    d = CudaDevice(0)
    yield d
    d.deinit()


@pytest.mark.parametrize("lens,clip", [((5, 3, 1), False), ((200001, 3), False), ((64,) * 50, False), ((5, 3, 1), True), ((200001, 3), True), ((64,) * 50, True)],
                         ids=lambda x: str(x[:2]) if isinstance(x, tuple) else "clip" if x else "plain")
def test_adam(fresh, lens, clip):
    n, g = sum(lens), rng(sum(lens))
    segs, off = [], 0
    for k in lens:
        segs.append((off, k))
        off += k
    p, gr, m, t = (g.standard_normal(n).astype(np.float32) for _ in range(4))
    v = g.random(n).astype(np.float32)
    P, G, M, V, T, N = (fresh.from_numpy(x) for x in (p, gr, m, v, t, np.zeros(len(segs), np.float32)))
    if clip:  # the norms' sums need work space: its first slot is there, the tickets' is not
        fresh.segment_sumsq(G, segs, N)
    count = fresh.from_numpy(np.array([11], np.uint64))
    fresh.capture.open()
    fresh.dispatch(opspec.adam(P, G, M, V, segs, 1, 1e-3, clip=clip, max_norm=0.5, norms=N, step_counter=count, soft_target=T, tau=0.25))
    fresh.capture.save()
    fresh.capture.run()
    want = OracleBackend().adam(p, gr, m, v, segs, 12, 1e-3, clip=clip, max_norm=0.5)
    for got, w in zip((P, G, M, V), want):
        assert rel_err(fresh.to_numpy(got), w) <= 1e-6
    assert rel_err(fresh.to_numpy(T), 0.25 * want[0] + 0.75 * t) <= 1e-6
    assert fresh.to_numpy(count)[0] == 11 + len(segs)
    fresh.capture.run()
    assert fresh.to_numpy(count)[0] == 11 + 2 * len(segs)



@pytest.mark.parametrize("rows,cols", [(5000, 33), (4099, 1003), (3000, 512), (70, 64)])
def test_column_sums_behind_an_op_that_left_work_space(fresh, rows, cols):
    x = rng(rows).standard_normal((rows, cols)).astype(np.float32)
    X, Y, S = fresh.from_numpy(x), fresh.from_numpy(np.zeros(cols, np.float32)), fresh.from_numpy(np.zeros(1, np.float32))
    fresh.dispatch(opspec.sum(X, S))
    fresh.capture.open()
    fresh.dispatch(opspec.unbroadcast(X, [rows, cols], Y, [cols], None, 1.0, 0.0))
    fresh.capture.save()
    for _ in range(2):
        fresh.capture.run()
        assert rel_err(fresh.to_numpy(Y), x.astype(np.float64).sum(0)) <= 1e-5
