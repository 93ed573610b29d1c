"""The autotuner times replayed step sequences, which is what runs after it: its time per
step is that of repeated calls under the shape it chose, for a small lattice and for a
batch of small lattices, where a launch or a graph's capture costs as much as the
steps.  (Both are device times of the same work; 30 % covers host noise.)"""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def replayed_ms(step, stream):
    """ms a step of repeated 16-step calls on this stream, best of five groups of three."""
    s = torch.cuda.ExternalStream(stream)
    best = 1e30
    for _ in range(3):
        step(16)
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(s)
        for _ in range(3):
            step(16)
        b.record(s)
        b.synchronize()
        best = min(best, a.elapsed_time(b) / 48)
    return best


def test_single_lattice(wt_lib):
    import windtunnel as wt
    e = wt.AeroEngine(dims=(64, 24, 20), origin=(wt.ORIGIN_X, 0.0, 0.0), h=0.18)
    e.set_shape_raw(wt.config_f1_shape(1))
    ms = min(e.tune()[2] for _ in range(3))

    def step(n):
        e.step(n, 0, 1.0)

    for _ in range(24):  # pending records at the start of a call: all sequences captured
        step(16)
    want = replayed_ms(step, e.stream())
    e.close()
    assert ms <= 1.3 * want, (ms, want)


@pytest.mark.parametrize("persist", ["0", "1"])
def test_batch(wt_lib, monkeypatch, persist):
    import windtunnel as wt
    monkeypatch.setenv("WT_BATCH_PERSIST", persist)
    grids = [((64, 36, 30), (wt.ORIGIN_X, 0.0, 0.0), 0.18)] * 12
    b = wt.AeroBatch(grids, wt.make_sim(storage="f16"))
    for e in b.lattices:
        e.set_shape_raw(wt.config_f1_shape(1))
    ms = min(b.tune()[2] for _ in range(3))
    want = replayed_ms(lambda n: b.step(n, 0, 1.0), b.stream())
    b.close()
    assert ms <= 1.3 * want, (ms, want)
