"""Tensor-core products of operands without 16-byte rows (odd leading dimensions, bases between words, batches), whose operands
are copied into the work space first, against a float64 product of the same operands.  bf16 inputs are exact in fp32 and
the sums of k products are fp32: 2e-5 of the largest element (5e-6 seen); fp32 inputs in three TF32 passes: 5e-5, as for
aligned ones."""
import sys
import threading

import numpy as np
import pytest

import oracle
from zigrad_b200 import opspec
from zigrad_b200.device import DeviceSlice

from .backends import GpuBackend
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


def between_words(be, a, off, bf16):
    """The array on the device, `off` elements past a 16-byte boundary."""
    pad = np.zeros(off, np.float32)
    x = np.concatenate([pad, a.ravel()])
    s = be.up((x.view(np.uint32) >> 16).astype(np.uint16), np.uint16) if bf16 else be.up(x)
    return DeviceSlice(s.ptr + off * s.itemsize, a.size, s.dtype, 0)


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("bf16,nb,m,n,k,off", [(True, 1, 300, 301, 501, 0), (True, 3, 129, 257, 263, 1), (True, 2, 2049, 513, 130, 7), (True, 1, 1000, 7, 2049, 3),
                                              (False, 1, 1023, 1001, 1001, 0), (False, 2, 701, 1024, 1003, 3),
                                              (False, 1, 300, 1025, 1001, 1), (False, 1, 250, 1025, 1001, 1), (False, 1, 163, 1429, 1194, 1)])
def test_operands_without_word_rows(gpu, bf16, nb, m, n, k, off, ta, tb):
    g, be = rng(m + n + k), GpuBackend(gpu)
    A, B = (g.standard_normal(s).astype(np.float32) for s in ((nb, k, m) if ta else (nb, m, k), (1, n, k) if tb else (1, k, n)))
    if bf16:
        A, B = (oracle.round_bf16(x.ravel()).reshape(x.shape) for x in (A, B))
    C0, bias = g.standard_normal((nb, m, n)).astype(np.float32), g.standard_normal(n).astype(np.float32)
    a, b = between_words(be, A, off, bf16), between_words(be, B, off, bf16)
    c = be.up(C0)
    gpu.dispatch(opspec.linear(a, b, c, m, n, k, ta, tb, m if ta else k, k if tb else n, n, 0.5, 2.0, "bias", be.up(bias), n_batch=(nb, 1, nb)))
    op = lambda x, t: (x.transpose(0, 2, 1) if t else x).astype(np.float64)
    want = 0.5 * (op(A, ta) @ op(B, tb)) + 2.0 * C0 + bias
    assert rel_err(be.down(c).reshape(nb, m, n), want) <= (2e-5 if bf16 else 5e-5)


def test_without_memory_for_the_copies(gpu):
    """The kernels that need no copies take over, and no error is left behind."""
    import torch
    g, be = rng(3), GpuBackend(gpu)
    m, n, k = 3001, 3003, 4001  # 48 MB of copies

    def product(m, n, k):
        A, B = (oracle.round_bf16(g.standard_normal(s).astype(np.float32).ravel()) for s in (m * k, n * k))
        return between_words(be, A, 1, True), between_words(be, B, 1, True), be.up(np.zeros((m, n), np.float32)), A.reshape(m, k), B.reshape(n, k)

    run = lambda a, b, c, m, n, k: gpu.dispatch(opspec.linear(a, b, c, m, n, k, False, True, k, k, n))
    for s in ((301, 301, 601), (3001, 3003, 41)):  # the kernels of both ways are loaded
        run(*product(*s)[:3], *s)
    a, b, c, A, B = product(m, n, k)
    gpu.sync()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (24 << 20), dtype=torch.uint8, device="cuda")
    try:
        run(a, b, c, m, n, k)
        gpu.sync()  # raises what was recorded
    finally:
        del hog
        torch.cuda.empty_cache()
    want = A[:64].astype(np.float64) @ B.T
    assert rel_err(be.down(c).reshape(m, n)[:64], want) <= 2e-5
    run(a, b, c, m, n, k)  # and the copies come back with the memory
    assert rel_err(be.down(c).reshape(m, n)[:64], want) <= 2e-5


@pytest.mark.parametrize("bf16", [True, False])
def test_two_threads_on_one_stream(gpu, bf16):
    """A product's copies are its own until it has been launched, whoever else issues products on the same stream.  (Without the
    lock that sees to it a copy of the other thread's has to fall into the few microseconds between two launches: rarely seen here.)"""
    g, be, m, n, k = rng(5), GpuBackend(gpu), 333, 1001, 1501
    jobs, wrong = [], []
    for _ in range(2):
        A, B = (g.standard_normal(s).astype(np.float32) for s in ((m, k), (n, k)))
        if bf16:
            A, B = (oracle.round_bf16(x.ravel()).reshape(x.shape) for x in (A, B))
        outs = [be.up(np.zeros((m, n), np.float32)) for _ in range(60)]
        jobs.append((between_words(be, A, 1, bf16), between_words(be, B, 1, bf16), outs, A.astype(np.float64) @ B.T.astype(np.float64)))
    start = threading.Barrier(2)

    def issue(a, b, outs):
        start.wait()
        for c in outs:
            gpu.dispatch(opspec.linear(a, b, c, m, n, k, False, True, k, k, n))

    was = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    threads = [threading.Thread(target=issue, args=j[:3]) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    sys.setswitchinterval(was)
    gpu.sync()
    for _, _, outs, want in jobs:
        wrong += [e for e in (rel_err(be.down(c).reshape(m, n), want) for c in outs) if e > 5e-5]
    assert not wrong, len(wrong)
