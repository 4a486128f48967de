"""Tile table files name the contraction levels they were measured for: one of an iteration of other levels (35 groups, as
written before) gives no entries, and a warning; the plan of a mixed handle has the levels that the files are checked for."""
import json

import pytest


def _write(path, entries, **more):
    path.write_text(json.dumps({"format": "", "note": "", "entries": entries, **more}))
    return str(path)


def test_tables_of_other_levels_are_not_used(tmp_path):
    from helios_gb300 import api
    ours = [[0, 0, 8, 33, 2], [2, 5, 19, 38, 2]]
    assert api.read_tile_table(_write(tmp_path / "a.json", ours)) == [tuple(e) for e in ours]
    assert api.read_tile_table(_write(tmp_path / "b.json", ours, levels=api.PLAN_LEVELS)) == [tuple(e) for e in ours]
    for path in (_write(tmp_path / "c.json", ours + [[0, 34, 8, 33, 1]]), _write(tmp_path / "d.json", ours, levels=7)):
        with pytest.warns(UserWarning, match="levels"):
            assert api.read_tile_table(path) == []
    api.write_tile_table(str(tmp_path / "e.json"), ours)
    assert json.loads((tmp_path / "e.json").read_text())["levels"] == api.PLAN_LEVELS
    assert len(api.read_tile_table(api.TILE_TABLE_PATH)) > 0


@pytest.mark.gpu
def test_levels_of_the_plan():
    from helios_gb300 import api, molecules
    cc = api.CoupledCluster(molecules.polyene(8), api.Keywords(precision="mixed"))
    assert cc.tile_choices()[0].shape == (4, api.PLAN_LEVELS)
    cc.finalizeCC()
