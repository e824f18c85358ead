"""The tuning that asks the wave engine for its grid form: told apart from the default, kept by other changes, refused for
ray casts, and saved and loaded with the autotuner's entries of frames and batches only."""
import pytest


def test_grid_always_is_not_the_default(R):
    ctx = R.Context(-1)
    assert ctx.tuning()["wave_refill"] == R.REFILL_GRID
    ctx.set_tuning(wave_refill=R.REFILL_GRID_ALWAYS)
    ctx.set_tuning(trace_block=256)
    t = ctx.tuning()
    assert t["wave_refill"] == R.REFILL_GRID_ALWAYS and t["trace_block"] == 256
    ctx.set_tuning(wave_refill=0)
    assert ctx.tuning()["wave_refill"] == R.REFILL_GRID
    with pytest.raises(R.ReinaError):
        ctx.set_tuning(refill=R.REFILL_GRID_ALWAYS)
    with pytest.raises(R.ReinaError):
        ctx.set_tuning(wave_refill=253)
    ctx.close()


@pytest.fixture
def own_ctx(R):
    """A context of the test's own: the cache of a shared one is saved by others."""
    c = R.Context(-1)
    yield c
    c.close()


def test_saved_entries(R, own_ctx, tmp_path):
    src, out = tmp_path / "in.txt", tmp_path / "out.txt"
    src.write_text("2 31 30 -1 64 16 0 1 2\n3 31 30 -1 128 12 1048576 1 2\n2 31 29 0 256 8 0 1 2\n")
    R.autotune_load(own_ctx, src)
    assert R.autotune_lookup(own_ctx, R.TUNE_RENDER, 1 << 31, 1 << 30)["wave_refill"] == R.REFILL_GRID_ALWAYS
    assert R.autotune_lookup(own_ctx, R.TUNE_BATCH, 1 << 31, 1 << 30)["wave_refill"] == R.REFILL_GRID_ALWAYS
    assert R.autotune_lookup(own_ctx, R.TUNE_RENDER, 1 << 31, 1 << 29)["wave_refill"] == R.REFILL_GRID
    R.autotune_save(own_ctx, out)
    assert "2 31 30 -1 64 16 0 1 2 0" in out.read_text().splitlines()


@pytest.mark.parametrize("line", ["0 20 21 -1 128 12 0 1 1", "1 20 21 -1 128 12 0 1 1", "2 20 21 -2 128 12 0 1 1", "3 20 21 33 128 12 0 1 1"])
def test_refused_entries(R, own_ctx, tmp_path, line):
    p = tmp_path / "bad.txt"
    p.write_text(line + "\n")
    with pytest.raises(R.ReinaError):
        R.autotune_load(own_ctx, p)


def test_paths_of_a_frames_entry(R, own_ctx, tmp_path):
    """A frame's entry keeps the paths it was timed with in the wave_paths column; as tuning it is no wave size."""
    src, out = tmp_path / "in.txt", tmp_path / "out.txt"
    src.write_text("2 10 12 8 128 12 65536 1 2\n3 10 12 8 128 12 65536 1 2\n")
    R.autotune_load(own_ctx, src)
    assert R.autotune_lookup(own_ctx, R.TUNE_RENDER, 1 << 10, 1 << 12)["wave_paths"] == R.DEFAULT_WAVE_PATHS
    assert R.autotune_lookup(own_ctx, R.TUNE_BATCH, 1 << 10, 1 << 12)["wave_paths"] == 65536
    R.autotune_save(own_ctx, out)
    assert "2 10 12 8 128 12 65536 1 2 0" in out.read_text().splitlines()
