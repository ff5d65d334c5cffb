"""Host logic of the SM shares two concurrent split-K weight gradients get (no GPU needed)."""
from zigrad_b200.mlp import shares_by_finish


def test_headline_step_shares():
    # 784-128 (7 output tiles) beside 128-64 (1 tile), batch 8192 = 256 k-slabs, 148 SMs:
    # 18 K ranges of 15 slabs for the first, 22 ranges of 12 slabs, four slabs' time later, for the second
    assert shares_by_finish(148, 7, 1, 256) == (126, 22)


def test_shares_never_exceed_the_gpu_and_keep_whole_tiles():
    for sms in (8, 64, 132, 148):
        for t0, t1 in ((7, 1), (1, 1), (4, 2), (13, 3)):
            for slabs in (4, 32, 256, 2048):
                got = shares_by_finish(sms, t0, t1, slabs)
                if got is None:
                    assert sms < t0 + t1
                    continue
                a, b = got
                assert a % t0 == 0 and b % t1 == 0 and a >= t0 and b >= t1 and a + b <= sms
                end = lambda a, b: max(-(-slabs // (a // t0)), -(-slabs // (b // t1)) + 4)
                for s0 in range(1, (sms - t1) // t0 + 1):  # no other split ends sooner
                    assert end(a, b) <= end(t0 * s0, (sms - t0 * s0) // t1 * t1)
