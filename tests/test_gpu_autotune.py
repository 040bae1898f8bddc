"""dsss_autotune runs every setting that makes a difference once: settings
that differ only in knobs without effect share a time, and those knobs keep
their defaults."""
import pytest

pytestmark = pytest.mark.gpu


def test_runs_each_distinct_setting_once(dsss, ctx):
    trials = 2
    ds = dsss.DeviceStrings(dsss.gen_dn(60000, 40, 20, seed=3))
    with dsss.tuned(sort_small_max=-1, sort_pivot=-1, sort_split_min=-1, sort_bits=-1, sort_seg_bits=-1):
        ctx.set_timing(True)
        t = dsss.autotune(ctx, ds, 4, trials=trials)
        runs = ctx.kernel_times()["stage:sort"][0]
        ctx.set_timing(False)
        assert runs == 3 * 2 * (1 + trials)
        assert t["settings_tried"] == 30
        for knob in ("sort_split_min", "sort_bits", "sort_seg_bits"):
            assert t[knob] == 0 and dsss.tune_get(knob) == 0
