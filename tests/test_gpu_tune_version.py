"""The autotuner's cache file outlives the library that wrote it: entries
timed with other kernels must not be found."""
import pytest

import shrinkage_full_tests_b200 as srk

pytestmark = pytest.mark.gpu


def test_entries_of_other_kernels_are_not_found(torch_cuda, tmp_path, monkeypatch):
    torch = torch_cuda
    N, e, B = 130, 16, 2  # N % 8 != 0, FP32: the FFT schedules are the only candidates
    W = N - 2 * e
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("SRK_TUNE_CACHE", str(cache))
    name = torch.cuda.get_device_name().replace(" ", "_")
    old = "%s:N%d:W%d:e%d:B%d:t0 512 0\n" % (name, N, W, e, B)
    cache.write_text(old)
    found = srk.autotune(N, W, e, 1.0, B)
    lines = cache.read_text().splitlines()
    assert lines[0] == old.strip() and len(lines) == 2  # the old entry stays, the configuration was timed anew
    assert lines[1].split(":")[0] == name and lines[1].split()[0] != lines[0].split()[0]
    assert srk.autotune(N, W, e, 1.0, B) == found
    assert cache.read_text().splitlines() == lines
