"""The 2-D acoustic tests of order 8 on the tiled kernels.

Their grids are small, so the library runs them on its small-grid kernels
(32 x 8 cells a CTA); here the same tests run with the 64 x 32 tiles of large
surveys asked for, so that strip formats, checkpoints, host tapes, segments,
illumination, free faces, per-shot models and shot groups meet both."""
import itertools

import pytest

import tests.test_acoustic2d_gpu as base
import tests.test_bench_geometry_gpu as bench
import tests.test_checkpoint_gpu as checkpoint
import tests.test_edge_cases_gpu as edge
import tests.test_free_surface_gpu as free
import tests.test_illumination_gpu as illumination
import tests.test_runner_gpu as runner
import tests.test_schedule_gpu as schedule
import tests.test_storage_gpu as storage
from tests.test_bench_geometry_gpu import many_oracle  # noqa: F401

pytestmark = pytest.mark.gpu

TESTS = [
    base.test_matches_reference_golden, base.test_matches_oracle, base.test_off_grid_receivers_record_zero,
    base.test_run_to_run_bit_exact, base.test_gradient_matches_central_differences,
    base.test_c2_geometry_against_oracle, base.test_wavelet_linearity,
    storage.test_fp32_baseline_matches_reference, storage.test_reduced_storage_matches_reference,
    storage.test_host_tape_is_bit_identical, checkpoint.test_acoustic2d_checkpoint,
    checkpoint.test_acoustic_recursive_checkpointing, illumination.test_matches_reference_and_oracle,
    illumination.test_illumination_does_not_move_the_gradient, illumination.test_does_not_depend_on_the_memory_mode,
    free.test_free_surface_matches_reference, free.test_free_surface_full_mode_and_storage_agree,
    free.test_per_face_free_surfaces_match_reference, runner.test_segments_equal_one_call,
    edge.test_acoustic2d_very_short_time_axes, edge.test_a_shot_with_every_receiver_off_the_grid,
    edge.test_sources_off_the_grid_give_zero_records_and_gradient,
    edge.test_acoustic2d_boxes_thinner_than_two_strips, schedule.test_graph_and_stream_launches_agree,
    schedule.test_shot_grouping_changes_no_result,
]


def _calls():
    """Every parameter set of a test that is a 2-D acoustic case."""
    for fn in TESTS:
        marks = [m for m in getattr(fn, "pytestmark", []) if m.name == "parametrize"]
        names = [[n.strip() for n in m.args[0].split(",")] for m in marks]
        for values in itertools.product(*[m.args[1] for m in marks]):
            kw = {}
            for ns, v in zip(names, values):
                kw.update(zip(ns, v if len(ns) > 1 else [v]))
            case = str(kw.get("case", kw.get("name", "acoustic2d")))
            if case.startswith("acoustic2d"):
                yield pytest.param(fn, kw, id="-".join([fn.__name__[5:], *map(str, kw.values())]))


@pytest.fixture
def tiled(monkeypatch):
    """Solvers made in the test ask for 32-row tiles; those made so."""
    import sweep_b200
    from sweep_b200 import autotune
    made = []

    class Tiled(sweep_b200.PropTorch):
        def __init__(self, equation, *args, schedule=None, **kw):
            if isinstance(equation, sweep_b200.Acoustic):
                schedule = dict(schedule or {}, tile_y=32)
                made.append(self)
            super().__init__(equation, *args, schedule=schedule, **kw)

    monkeypatch.setattr(sweep_b200, "PropTorch", Tiled)
    autotune.clear_schedules()
    yield made
    autotune.clear_schedules()


@pytest.mark.parametrize("fn,kw", list(_calls()))
def test_on_tiles(fn, kw, tiled):
    fn(**kw)
    assert tiled


@pytest.mark.parametrize("fwd,rev", [(2, 8), (4, 16), (1, 1)])
def test_shot_groups_on_tiles(fwd, rev, many_oracle, tiled):  # noqa: F811
    bench.test_acoustic2d_shot_groups_match_reference(fwd, rev, many_oracle)
    assert tiled
