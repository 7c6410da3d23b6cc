"""The tuner measures tile heights only where they can differ."""
from fmm_gen_b200 import tuner


def test_no_tile_trials_for_a_measurement_whose_heights_run_alike():
    calls = []

    def measure(choices, tiles=None):
        calls.append(tiles)
        return 100.0 - (1.0 if tiles else 0.0)  # noise that the refinement would take for a gain

    shapes = [(256, 256, 4096)] * 2 + [(2048, 2048, 512)] * 6
    measure.tile_heights = False
    rep = tuner.BatchTuner().tune(shapes, measure)
    assert all(t is None for t in calls)
    assert set(rep.tiles) == {tuner.TILE} and all("64-row" not in name for name, _ in rep.trials)


def test_the_library_measurement_says_so():
    assert tuner.batch_timer(None, [], [], [], []).tile_heights is False
