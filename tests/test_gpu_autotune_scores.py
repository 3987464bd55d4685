"""Rates the autotuner measures for scorings whose calibration pairs could
score more than the lanes hold: a class's time per cell does not depend on
the scores, so they have to be those of a scoring with small ones (same
lanes), and nothing of the calibration may be rerun.
"""
import pytest

import ipuma_b200 as ib

pytestmark = pytest.mark.gpu


def _rates(forward_only, gap_init, gap_extend, match, mismatch):
    with ib.Engine(ib.sw_config(gap_init, gap_extend, match, mismatch, mismatch),
                   ib.algo_config(forward_only=forward_only)) as e:
        e.autotune()
        return {(c["lanes"], c["k"]): c["slot_ps"] for c in e.tuning()["classes"]}


# gap_init, gap_extend, match, mismatch; rates are kept by the gaps, so the
# two scorings of a row have different ones.
@pytest.mark.parametrize("forward_only", [True, False])
@pytest.mark.parametrize("high,low", [((-7, -3, 50, -40), (-8, -3, 32, -26)),   # unscaled lanes
                                      ((-7, -2, 110, -90), (-8, -2, 32, -26)),  # the largest that run in lanes
                                      ((0, -1, 5, -4), (0, -2, 1, -1))])        # linear gaps
def test_high_scores_do_not_shorten_the_calibration(high, low, forward_only):
    a, b = _rates(forward_only, *high), _rates(forward_only, *low)
    for lanes, k in ((16, 8), (16, 16), (32, 12), (32, 16)):
        # A third: what two measurements of one class have been seen to
        # differ by is below a tenth; a class that gives up half way reads
        # as half its time or less.
        assert 0.67 < a[lanes, k] / b[lanes, k] < 1.5, (lanes, k, a, b)
