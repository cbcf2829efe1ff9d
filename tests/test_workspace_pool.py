"""Whose scratch a drop-in call works on: never that of another stream, another host thread or a captured graph."""

import threading

import pytest
import torch

from nki_library_b200 import _lib, pipeline


class _Fake:
    def __init__(self, *shape, zeroed=True):
        self.shape, self.zeroed = shape, zeroed


@pytest.fixture
def pool(monkeypatch):
    """``get(shape, stream, capturing)`` on a machine without a GPU."""
    now = {}
    monkeypatch.setattr(_lib, "stream_ptr", lambda: now["stream"])
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: now["capturing"])
    monkeypatch.setattr(pipeline, "BlockWorkspace", _Fake)
    monkeypatch.setattr(pipeline, "DenseWorkspace", _Fake)

    def get(kind, shape, stream=7, capturing=False):
        now.update(stream=stream, capturing=capturing)
        fn = pipeline.get_workspace if kind == "mx" else pipeline.get_dense_workspace
        return fn(*shape, torch.device("cuda", 0))

    return get


@pytest.mark.parametrize("kind", ["mx", "dense"])
def test_streams_threads_and_captures_do_not_share(pool, kind):
    a = (128, 256, 512)
    first = pool(kind, a)
    assert pool(kind, a) is first
    assert pool(kind, a, stream=8) is not first
    assert pool(kind, a) is first and pool(kind, a, stream=8) is pool(kind, a, stream=8)
    other = []
    t = threading.Thread(target=lambda: other.append(pool(kind, a)))
    t.start()
    t.join()
    assert other[0] is not first
    graph = pool(kind, a, capturing=True)
    assert graph is not first and not graph.zeroed  # a captured fill would run in every replay
    assert pool(kind, a, capturing=True) is not graph and pool(kind, a) is first


@pytest.mark.parametrize("kind", ["mx", "dense"])
def test_only_the_oldest_is_dropped(pool, kind):
    shapes = [(128 * i, 256, 1024) for i in range(1, 7)]
    held = [pool(kind, s) for s in shapes[:5]]
    assert pool(kind, shapes[0]) is held[0]  # now the youngest
    pool(kind, shapes[5])                    # drops shape 1
    for i in (0, 2, 3, 4):
        assert pool(kind, shapes[i]) is held[i]
    assert pool(kind, shapes[1]) is not held[1]


def _moe(T, seed, E=16, K=2, H=1024, I=512):
    import nki_library_b200 as m
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((T, H), device="cuda", generator=g).to(torch.bfloat16)
    aff = torch.rand((T, E), device="cuda", generator=g)
    idx = aff.topk(K, dim=1).indices.to(torch.int32)
    return lambda w: m.moe_tkg(x, w, None, aff, idx, False,
                               expert_affinities_scaling_mode=m.ExpertAffinityScaleMode.POST_SCALE)


@pytest.fixture(scope="module")
def weights():
    from nki_library_b200.layer import random_expert_weights
    return random_expert_weights(16, 1024, 512, "cuda", seed=4)


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [False, True])
def test_equal_shapes_on_two_streams(weights, threads):
    calls = [_moe(64, 1), _moe(64, 2)]
    ref = [c(weights).clone() for c in calls]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[], []]

    def work(i, n):
        with torch.cuda.stream(streams[i]):
            for _ in range(n):
                got[i].append(calls[i](weights))

    if threads:
        ts = [threading.Thread(target=work, args=(i, 40)) for i in range(2)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    else:
        for _ in range(40):
            work(0, 1)
            work(1, 1)
    torch.cuda.synchronize()
    for i in range(2):
        assert all(torch.equal(o, ref[i]) for o in got[i])


@pytest.mark.gpu
def test_captured_call_outlives_the_pool(weights):
    call = _moe(64, 3)
    ref = call(weights).clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call(weights)
    for T in (1, 2, 3, 4, 5, 6, 7, 8, 100):  # other shapes push everything else out of the pool
        _moe(T, T)(weights)
    torch.cuda.synchronize()
    marks = [torch.full((n,), 77, dtype=torch.uint8, device="cuda") for n in (1 << 20, 1 << 22, 1 << 24) for _ in range(8)]
    for _ in range(3):
        graph.replay()
        _moe(64, 5)(weights)
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
    assert all(bool((t == 77).all()) for t in marks)
