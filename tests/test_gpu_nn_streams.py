"""Bias gradients and losses of different inputs in flight on several streams at once,
from one thread and from several, give the bits that the calls give one after another."""
import threading

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SIZES = [(200003, 16), (40001, 64), (300007, 8), (70001, 128)]


@pytest.fixture(scope="module")
def work(wt_lib):
    from windtunnel.net import Ops
    ops = Ops()
    g = torch.Generator(device="cuda").manual_seed(1)
    jobs = []
    for rows, c in SIZES:
        dy = torch.randn((rows, c), generator=g, device="cuda").to(torch.bfloat16)
        pred, target = torch.randn((rows, 8), generator=g, device="cuda").to(torch.bfloat16), torch.randn((rows, 4), generator=g, device="cuda")
        jobs.append((dy, pred, target))
    want = [run(ops, job, 1)[0] for job in jobs]
    torch.cuda.synchronize()
    return ops, jobs, want


def run(ops, job, times):
    dy, pred, target = job
    out = []
    for _ in range(times):
        db, loss, dpred = torch.zeros(dy.shape[1], device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda"), torch.empty_like(pred)
        ops.bias_grad(dy, db)
        ops.mse(pred, target, None, 3.0, dpred, loss)
        out.append((db, loss, dpred))
    return out


def same(got, want):
    return all(torch.equal(a, b) for a, b in zip(got, want))


def test_streams_of_one_thread(work):
    ops, jobs, want = work
    streams = [torch.cuda.Stream() for _ in jobs]
    got = [[] for _ in jobs]
    for _ in range(40):
        for k, (job, st) in enumerate(zip(jobs, streams)):
            with torch.cuda.stream(st):
                got[k] += run(ops, job, 1)
    torch.cuda.synchronize()
    assert all(same(r, w) for rs, w in zip(got, want) for r in rs)


def test_threads(work):
    ops, jobs, want = work
    got = [None] * len(jobs)

    def one(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            got[k] = run(ops, jobs[k], 40)

    threads = [threading.Thread(target=one, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert all(same(r, w) for rs, w in zip(got, want) for r in rs)


def test_more_streams_than_keep_a_buffer(work):
    ops, jobs, want = work
    streams = [torch.cuda.Stream() for _ in range(24)]
    got = []
    for _ in range(4):
        for k, st in enumerate(streams):
            with torch.cuda.stream(st):
                got.append((k % len(jobs), run(ops, jobs[k % len(jobs)], 1)[0]))
    torch.cuda.synchronize()
    assert all(same(r, want[k]) for k, r in got)


def test_threads_of_one_stream(work):
    ops, jobs, want = work
    stream = torch.cuda.Stream()
    got = [None] * len(jobs)

    def one(k):
        with torch.cuda.stream(stream):
            got[k] = run(ops, jobs[k], 40)

    threads = [threading.Thread(target=one, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert all(same(r, w) for rs, w in zip(got, want) for r in rs)


def test_captured_calls_replay(work):
    """In a captured graph the scratch belongs to the graph."""
    ops, jobs, want = work
    dy, pred, target = jobs[0]
    db, loss, dpred = torch.zeros(dy.shape[1], device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda"), torch.empty_like(pred)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.bias_grad(dy, db)
        ops.mse(pred, target, None, 3.0, dpred, loss)
    for _ in range(3):
        db.zero_()
        loss.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert same((db, loss, dpred), want[0])
