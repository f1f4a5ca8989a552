"""The launch tunings that are tried differ in effect."""
from hashpoint import batch, native


def test_heavy_windows_tried_are_in_effect():
    native.build()
    held = min(native.stage_config_info(c)["stage_points"] // 16 for c in native.STAGE_CONFIGS)
    assert len(set(batch.Autotuner.HEAVY)) == len(batch.Autotuner.HEAVY) and max(batch.Autotuner.HEAVY) <= held
