"""CPU test of the generated table of quadrature points: another generator makes it anew."""
import importlib.util
import os
import sys

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gbasis_b200", "csrc")
sys.path.insert(0, CSRC)


def _generator(path, source, value):
    """gen_rys from changed source, its tables replaced by one number."""
    path.write_text(source)
    spec = importlib.util.spec_from_file_location(path.stem, path)
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    m.calls = []
    m.root_table = lambda n: m.calls.append(n) or [value]
    return m


def test_the_table_follows_its_generator(tmp_path):
    with open(os.path.join(CSRC, "gen_rys.py")) as f:
        source = f.read()
    assert "for _ in range(4):" in source  # Newton steps of the points
    one = _generator(tmp_path / "rys_one.py", source, 1.0)
    two = _generator(tmp_path / "rys_two.py", source.replace("for _ in range(4):", "for _ in range(5):"), 2.0)
    table = tmp_path / "rys_tables.cu"
    one.emit_sources(str(tmp_path), [(2, 1, 1, 1)])
    assert (1.0).hex() in table.read_text() and one.calls
    one.calls.clear()
    before = os.stat(table).st_mtime_ns
    one.emit_sources(str(tmp_path), [(2, 1, 1, 1)])  # nothing changed: neither made nor written again
    assert not one.calls and os.stat(table).st_mtime_ns == before
    two.emit_sources(str(tmp_path), [(2, 1, 1, 1)])
    assert (2.0).hex() in table.read_text() and (1.0).hex() not in table.read_text()
