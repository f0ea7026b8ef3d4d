"""The autotuner's cache and candidates."""
import pytest

from ems_b200 import gpu, synth

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("need_gpu")]


def test_cache_of_another_build_is_not_used(tmp_path, monkeypatch):
    """A line of the same window and GPU whose key has another build's name, or
    none as older libraries wrote it, is not taken."""
    path = tmp_path / "tuning.txt"
    monkeypatch.setenv("SHOC_TR_TUNE_CACHE", str(path))
    case = synth.make("small")

    def tuned():
        t = gpu.TracerStep(case)
        t.start()
        best, cached = t.autotune_ex(1)
        t.close()
        return cached

    assert not tuned()
    assert tuned()
    key, values = path.read_text().split(None, 1)
    window = key.split("|")[-13:]  # GPU model and window configuration
    path.write_text("".join("%s %s" % ("|".join(head + window), values)
                            for head in (["v2"], ["v3", "0" * 12])))
    assert not tuned()


@pytest.mark.parametrize("precision", [gpu.FP64, gpu.FP32_MIXED])
def test_launches_that_are_the_same_are_tried_once(precision):
    """Two tracers: two warps per block, whatever more is asked for; FP32-mixed with
    and without the prefetch (the fused kernel does not take so many layers)."""
    case = synth.build_case("tune", 40, 30, synth.uniform_layers(120, 600.0), seed=9, ntr=2,
                            depth=(500.0, 599.0))
    t = gpu.TracerStep(case, precision=precision)
    t.start()
    t.run(3)
    t.sync()
    n = t.launches()
    t.run(1)
    t.sync()
    step, n = t.launches() - n, t.launches()
    t.autotune(1)
    most = {gpu.FP64: 1, gpu.FP32_MIXED: 2}[precision]
    assert t.launches() - n <= most * step
    t.close()
