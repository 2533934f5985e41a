"""What the choice of threads per subset (csrc/icgn_tile.cu) depends on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [64, 128, 256])
@pytest.mark.parametrize("n", [1, 100, 500])
def test_a_tuned_choice_holds_for_small_batches(gpv_mod, tmp_path, monkeypatch, threads, n):
    """A context's tuned threads (here from its cache file) are used for every batch
    of the class, those of one subset per SM and less too: the bytes are those of the
    same threads by GPV_TILE_THREADS."""
    import torch
    from gpv import synth
    W = synth.workload(3, scale_down=4)
    side = W["f"].shape[0]
    rng = np.random.default_rng(threads + n)
    xy = rng.uniform(33, side - 33, (n, 2))
    d = gpv_mod.make_desc(xy, 25, 1, synth.seeded_p0(W["field"], xy, rng, 0.2))
    d["p0"][:, 6:] = 0.0

    def solve():
        ctx = gpv_mod.Context(0)
        F, G = gpv_mod.Image(image_gs=W["f"], ctx=ctx), gpv_mod.Image(image_gs=W["g"], ctx=ctx)
        return gpv_mod.solve_batch(F, G, d).tobytes()

    monkeypatch.setenv("GPV_TILE_THREADS", str(threads))
    want = solve()
    monkeypatch.delenv("GPV_TILE_THREADS")
    cache = tmp_path / "tune.txt"
    cache.write_text(f"{torch.cuda.get_device_name(0)}|1|{threads}|-1|4\n")
    monkeypatch.setenv("GPV_TUNE_CACHE", str(cache))
    assert solve() == want


@pytest.mark.parametrize("line,want", [("|0|64|-1|8", 4), ("|0|64|-1|4", 4), ("|0|128|2|0", 0), ("|0|128|2", 0), ("|0|128", 0)])
def test_cached_run_lengths_are_the_ones_solved_with(gpv_mod, tmp_path, monkeypatch, line, want):
    """Cache lines of run length 8, which no kernel has any more, are reported as
    what they run as."""
    import torch
    cache = tmp_path / "tune.txt"
    cache.write_text(torch.cuda.get_device_name(0) + line + "\n")
    monkeypatch.setenv("GPV_TUNE_CACHE", str(cache))
    ctx = gpv_mod.Context(0)
    assert (ctx.tuning()[0]["run_length"] or 0) == want
