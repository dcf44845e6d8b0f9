"""The batch autotuner's candidates and its sample of a batch (no GPU)."""

from __future__ import annotations

import pytest

from planet_renderer_gb300.atmosphere import autotune
from planet_renderer_gb300.atmosphere.batch import AERIAL, Tuning
from planet_renderer_gb300.atmosphere.workloads import batched_lut_jobs


def test_candidates_are_distinct_launches():
    """Item sizes are rounded up to multiples of 32: no two candidates are the same then."""

    def effective(t: Tuning):
        return tuple(-(-v // 32) * 32 for v in (t.sky_view_texels_per_item, t.aerial_columns_per_item)) + (t.blocks_per_sm,)

    assert len({effective(t) for t in autotune.CANDIDATES}) == len(autotune.CANDIDATES) > 1
    for t in autotune.CANDIDATES:
        assert 1 <= min(effective(t)[:2]) and max(effective(t)[:2]) <= 4096 and 1 <= t.blocks_per_sm <= 8


@pytest.mark.parametrize("snapshots,cameras", [(1, 1), (1, 8), (2, 8), (8, 8), (16, 8)])
def test_sample_is_split_as_the_batch_is(snapshots, cameras):
    jobs = batched_lut_jobs(2027, snapshots, cameras)

    def columns(some):
        return sum(j.width * j.height for j in some if j.kind == AERIAL)

    line = 256 * 3 * 152 / 4
    part = autotune.sample(jobs, 8, 152)
    assert 0 < len(part) <= len(jobs) and (columns(part) <= line) == (columns(jobs) <= line)
    if columns(jobs) <= line or columns(jobs[::8]) > line:
        assert part == jobs[::8]
