"""Option 'merge_launches': consecutive stencil groups without a hazard run
as one launch.  Every run's members are pairwise independent, the launch
list keeps every order, and the launch count drops by the members merged
away."""

import re

import pytest

from polymage_b200 import codegen
from polymage_b200.apps import catalog


@pytest.mark.parametrize("name", ["pyramid8", "pyramid", "laplacian"])
def test_merged_launches_are_independent(name, monkeypatch):
    seen = {}
    plan = codegen.plan_merges

    def record(pg, pipeline):
        runs = plan(pg, pipeline)
        seen.update(runs=runs, rw=list(pg.launch_rw))
        return runs
    monkeypatch.setattr(codegen, "plan_merges", record)
    drop = ('merge_launches',)
    alone = catalog.variant(name, drop_options=drop).generate_code()
    mod = catalog.variant(name, ('merge_launches',), drop).generate_code()
    runs, rw = seen["runs"], seen["rw"]
    assert runs and all(len(r) > 1 for r in runs)
    for run in runs:
        assert run == list(range(run[0], run[-1] + 1))
        for a in run:
            for b in run:
                if a < b:
                    assert not rw[a][1] & rw[b][0]
                    assert not rw[a][0] & rw[b][1]
                    assert not rw[a][1] & rw[b][1]
    merged = sum(len(r) - 1 for r in runs)
    assert mod.meta['launches'] == alone.meta['launches'] - merged
    body = mod.source[mod.source.index("static int pm_run("):]
    body = body[:body.index("\n}\n")]
    calls = re.findall(r"launch_(pm_\w+)\(A", body)
    assert len(calls) == mod.meta['launches']
    assert sum("merge" in c for c in calls) == len(runs)


def test_a_dependent_group_is_not_merged():
    """Harris in groups of three stages: each group reads the one before."""
    from polymage_b200.apps.harris import build_harris
    p = build_harris(tile_sizes=(32, 64), group_size=3,
                     options=('merge_launches',))
    mod = p.generate_code()
    for run in mod.meta.get('merges', []):
        assert len(run) > 1
    assert mod.meta['launches'] <= len(p.groups)
