"""CPU tests of the tuning cache: a file measured on other kernels changes nothing."""
import json

import pytest

from gbasis_b200 import autotune
from gbasis_b200.batch import EriBatch


class _Fake:
    """A basis or batch of three blocks that records the knobs set on it."""

    def __init__(self):
        self.calls = []

    def blocks(self):
        return [((0, 0, 0, 0), 4, 128.0, 10), ((2, 1, 2, 0), 1, 16.0, 10), ((3, 3, 3, 3), 1, 1.0, 2)]

    types = blocks

    def set_team(self, k, team):
        self.calls.append(("team", k, team))

    def set_block_config(self, k, variant, ctas):
        self.calls.append(("config", k, variant, ctas))

    set_type_config = set_block_config

    def set_streams(self, n):
        self.calls.append(("streams", n))


TABLE = {"0000:7": 32, "v:2120:4": 1, "v:3333:0": 1, "c:0000:7": 2, "streams": 1}
EXPECTED = [("team", 0, 32), ("config", 0, 0, 2), ("config", 1, 1, 8), ("config", 2, 1, 8)]


def _both():
    basis, batch = _Fake(), _Fake()
    autotune.apply_cache(basis)
    EriBatch.apply_tuning(batch)
    return basis.calls, batch.calls


@pytest.fixture
def cache(tmp_path, monkeypatch):
    path = tmp_path / "tuning.json"
    monkeypatch.setenv("GBX_TUNE_CACHE", str(path))
    return path


@pytest.mark.parametrize("tag", [{}, {"kernels": autotune.KERNELS - 1}, {"kernels": None}])
def test_a_file_of_other_kernels_changes_nothing(cache, tag):
    cache.write_text(json.dumps({**TABLE, **tag}))
    assert _both() == ([], [])


def test_stored_choices_are_applied(cache):
    """Choices go into a file of this generation and come back; an older file's entries do not
    survive under the new tag."""
    cache.write_text(json.dumps({"1111:7": 8}))
    autotune._store(TABLE)
    assert json.loads(cache.read_text()) == {**TABLE, "kernels": autotune.KERNELS}
    assert _both() == (EXPECTED + [("streams", 1)], EXPECTED)
    autotune._store({"streams": 3})
    assert autotune._load() == {**TABLE, "streams": 3}


def test_defaults_are_not_stored(cache):
    autotune._store(TABLE)
    autotune._store({"v:2120:4": 0, "c:0000:7": 8, "v:3333:0": 2, "0000:7": 16})
    assert autotune._load() == {"0000:7": 16, "v:3333:0": 2, "streams": 1}


@pytest.mark.parametrize("times,pick", [((9.0, 8.9, 9.5), 2), ((9.0, 8.0, 9.5), 4), ((7.0, 7.1, 9.5), 2),
                                        ((9.0, 9.0, 1.0), 8)])
def test_a_knob_moves_for_a_clear_gain_only(times, pick):
    assert autotune._pick((2, 4, 8), times, 2) == pick
    assert autotune._pick((4, 8), times[1:], 2) == (4, 8)[times[2] < times[1]]


@pytest.mark.parametrize("entry,team,quartets,lanes", [
    (2, 16, 10, 16), (2, 16, 1200, 16), (2, 16, 2368, 16), (2, 16, 4736, 8), (2, 16, 9472, 4),
    (2, 16, 18944, 2), (1, 4, 37887, 2), (1, 4, 37888, 1), (32, 16, 10, 32), (32, 16, 591, 32),
    (32, 16, 592, 16), (8, 8, 10, 8), (8, 8, 10 ** 6, 8)])
def test_short_lists_keep_the_lanes_that_fill_the_device(entry, team, quartets, lanes):
    assert autotune._lanes(entry, team, quartets) == lanes


def test_the_shipped_file_belongs_to_these_kernels(monkeypatch):
    monkeypatch.delenv("GBX_TUNE_CACHE", raising=False)
    assert autotune._load()


def test_a_table_of_the_caller_is_used_as_it_is(cache):
    basis, batch = _Fake(), _Fake()
    autotune.apply_cache(basis, TABLE)
    EriBatch.apply_tuning(batch, TABLE)
    assert (basis.calls, batch.calls) == (EXPECTED + [("streams", 1)], EXPECTED)
