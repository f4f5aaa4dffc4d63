"""The tuner tries the streaming kernels' knobs where those kernels run: grids
that go by point have only the steps per graph to choose."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,stream", [((24, 20, 18), False), ((3, 20, 18), True),
                                          ((96, 96, 120), True)])
def test_candidates_that_act(gpu_lib, tmp_path, monkeypatch, shape, stream):
    from nlsemagic_gb300 import autotune
    monkeypatch.setenv("NLSE_TUNE_CACHE", str(tmp_path / "tune.json"))
    entry = autotune.tune(shape, method=2, precision=3, BC=2, steps=2)
    every = autotune.candidates(shape, 3)
    want = len(every) if stream else len({c["graph.steps"] for c in every})
    assert entry["candidates"] == 1 + want
    if not stream:
        assert (entry["wide.zc"], entry["wide.ty"]) == (0, 8)
