"""Boxes whose radii go to one launch of each pair pass are not tuned: no
timings, nothing in the cache; a number of radii that the caller fixed is."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [16, 64])
def test_small_boxes_are_not_tuned(hii, tmp_path, monkeypatch, N):
    cache = tmp_path / "tune.jsonl"
    monkeypatch.setenv("SF21_TUNE_CACHE", str(cache))
    fb = hii.FilterBank(N, 40.0, 0.7, [(30.0, 10.0, 8)])
    path, ms = fb.path()
    fb.close()
    assert path == 5 and not any(ms.values()) and not cache.exists()
    if N == 64:
        fb = hii.FilterBank(N, 40.0, 0.7, [(30.0, 10.0, 8)], kmax=8)
        path, ms = fb.path()
        fb.close()
        assert path in ms and all(ms[p] > 0 for p in (1, 5)) and len(cache.read_text().splitlines()) == 1
