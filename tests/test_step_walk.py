"""The walk a propagation takes by default (gpop_step_walk, what launch_gj8 asks): its bands by objects per SM, degree
and precision, and what its launches rely on for any GPU. Host arithmetic only: runs without a GPU."""
import pytest

SMS = 148


def test_bands():
    import opengpop_b200 as G
    # degree: last objects per SM of the teams, then of the column walk in FP64 and mixed precision
    for degree, team, cols64, cols_mixed in ((2, 64, 0, 0), (13, 64, 0, 0), (14, 32, 64, 128), (27, 32, 64, 128),
                                             (28, 24, 224, 224), (42, 24, 224, 224), (43, 8, 320, 256),
                                             (59, 8, 320, 256), (60, 4, 384, 320), (70, 4, 384, 320)):
        for prec, cols in ((G.FP64, cols64), (G.MIXED, cols_mixed)):
            W = lambda k, extra=0: G.step_walk(k * SMS + extra, SMS, prec, degree)
            assert W(0, 1)[0] == 3 and W(team)[0] == 3
            above = W(team, 1)[0]
            if cols:
                assert above == 6 and W(cols)[0] == 6
            beyond = W(max(cols, team), 1)[0]
            assert beyond in (1, 2, 5) and beyond != 6
            assert W(448, 1)[0] == 5  # the SM's last set of 64: plain blocks
            assert W(600)[0] == 5  # more than one wave
    # one object per thread: FP64 above the columns, and low degrees in both
    assert G.step_walk(256 * SMS, SMS, G.FP64, 36) == (1, 1, True)
    assert G.step_walk(256 * SMS + 1, SMS, G.FP64, 36)[0] == 2
    assert G.step_walk(128 * SMS + 1, SMS, G.MIXED, 20) == (1, 1, False)
    assert G.step_walk(256 * SMS, SMS, G.MIXED, 36) == (2, 1, False)
    assert G.step_walk(65536, SMS, G.MIXED) == (2, 1, False) and G.step_walk(65536, SMS, G.FP64) == (2, 1, True)


def test_teams():
    import opengpop_b200 as G
    for prec in (G.FP64, G.MIXED):
        # whole warps with a lane per column up to two objects per SM, the FP64 table up to four
        for degree, lanes in ((31, 32), (32, 64), (63, 64), (64, 96), (70, 96)):
            assert G.step_walk(1, SMS, prec, degree) == (3, lanes, True)
            assert G.step_walk(2 * SMS, SMS, prec, degree)[1] == lanes
        assert G.step_walk(4 * SMS, SMS, prec, 70) == (3, 32, True)
        assert G.step_walk(4 * SMS + 1, SMS, prec, 50)[2] == (prec == G.FP64)
    assert G.step_walk(8 * SMS, SMS, G.FP64, 50) == (3, 16, True)
    assert G.step_walk(7 * SMS, SMS, G.FP64, 20) == (3, 8, True)
    assert G.step_walk(64 * SMS, SMS, G.FP64, 8) == (3, 4, True)


@pytest.mark.parametrize("sms", [1, 7, 132, 148, 160])
def test_invariants(sms):
    import opengpop_b200 as G
    for prec in (G.FP64, G.MIXED):
        for degree in (2, 8, 9, 14, 20, 36, 50, 70):
            for n in list(range(1, 40 * sms, max(1, sms // 3))) + list(range(40 * sms, 700 * sms, 9 * sms + 1)):
                w, lanes, fp64 = G.step_walk(n, sms, prec, degree)
                assert w in (1, 2, 3, 5, 6) and (fp64 or prec == G.MIXED)
                if w == 3:  # a group fits a block of 256; within a warp a power of two, else a lane per column
                    assert lanes <= 256 and (lanes & (lanes - 1) == 0 if lanes <= 32 else
                                             lanes % 32 == 0 and lanes > degree)
                else:
                    assert lanes == 1
                if w == 6:
                    assert n <= 512 * sms and degree >= 14
                if w in (1, 2):
                    assert n <= 512 * sms


def test_rejects_bad_arguments():
    import opengpop_b200 as G
    for args in ((0, SMS, G.FP64, 70), (10, 0, G.FP64, 70), (10, SMS, 7, 70), (10, SMS, G.FP64, -1)):
        with pytest.raises(G.GpopError):
            G.step_walk(*args)
