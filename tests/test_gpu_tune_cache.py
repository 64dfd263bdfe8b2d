"""Lines of a tune file that were timed among other passes are not applied to new
fields, and a line written now is."""
import pytest

import qaxions_b200 as qx

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _fresh_tune_cache():
    qx.clear_tune_cache()
    yield
    qx.clear_tune_cache()


# without a generation, of another one, cut off
OLD = ["0 8 8 1 0 2 1 0 0.0489", "0 8 8 1 0 2 1 0 0.0489 : 1", "0 8 8 1 0 2 1 0 0.0489 :"]


@pytest.mark.parametrize("values", OLD)
def test_lines_of_other_passes_are_not_used(tmp_path, monkeypatch, values):
    path = tmp_path / "tune.txt"
    path.write_text(f"v3 3 96 c64 1 : {values}\n")
    monkeypatch.setenv("QX_TUNE_CACHE", str(path))
    with qx.Field(3, 96, dtype="c64", dt=1e-5) as f:
        t = f.get_tune()
        assert t["from_cache"] == 0 and t["plan"] == 0


def test_a_line_written_now_is_used(tmp_path, monkeypatch):
    path = tmp_path / "tune.txt"
    path.write_text("v3 2 16 c64 1 : 0 8 8 1 0 2 0 0 0.01\n")
    with qx.Field(2, 16, dtype="c64", dt=1e-5) as f:
        f.ic_config(qx.IC_GRF, 3, 0)
        ms, cached = f.autotune(1, cache=str(path))
        assert not cached and len(path.read_text().splitlines()) == 2
        chosen = f.get_tune()
    qx.clear_tune_cache()
    monkeypatch.setenv("QX_TUNE_CACHE", str(path))
    with qx.Field(2, 16, dtype="c64", dt=1e-5) as f:
        t = f.get_tune()
        assert t.pop("from_cache") == 1
        chosen.pop("from_cache")
        assert t == chosen
        ms2, cached = f.autotune(1, cache=str(path))
        assert cached and ms2 == pytest.approx(ms, rel=1e-5)
