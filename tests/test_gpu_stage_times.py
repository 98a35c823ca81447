"""Stage times account for a whole refine: over several waves and eight bounces
(nine rounds of extend, sort, light sampling, shade and shadow each) their sum
is the refine's device time."""
import pytest

from oxideav_render_b200 import abi, api, testscenes as ts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sort", [True, False])
@pytest.mark.parametrize("schedule,bounces,waves", [(abi.PT_SCHEDULE_WAVEFRONT, 8, 1), (abi.PT_SCHEDULE_WAVEFRONT, 8, 7),
                                                    (abi.PT_SCHEDULE_WAVEFRONT, 1, 5), (abi.PT_SCHEDULE_MEGAKERNEL, 8, 3)])
def test_stage_times_sum_to_the_device_time(schedule, bounces, waves, sort):
    c = api.Context(0)
    try:
        c.set_schedule(schedule)
        c.set_material_sort(sort)
        c.set_wave_slots(256 * 256)
        c.set_stage_timing(True)
        t = api.PathTracer(c)
        t.sync(ts.sphere_grid_c1(256, 1)[0], ts.pt_opts(256, waves, bounces, ambient=0.3))
        for _ in range(2):  # the second finds every kernel loaded
            t.refine(waves)
        assert api.batch_counters(c)["waves"] == waves
        # The refine's own events lie around the stages', with one upload of
        # the first wave's descriptor between the first of either: a few
        # microseconds of at least 400 (a wave of 64 K paths). A missing
        # stage of the last bounce alone is 10.
        total, parts = t.last_kernel_ms(), sum(t.stage_ms().values())
        assert 0.95 * total <= parts <= 1.001 * total
        t.close()
    finally:
        c.close()
