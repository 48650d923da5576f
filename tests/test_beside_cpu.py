"""The second stream of a step (`ops.beside`): what it leaves behind, with stand-ins for the streams."""

from __future__ import annotations

import contextlib
import threading
from types import SimpleNamespace

import pytest
import torch

from liteinfer_b200 import ops
from liteinfer_b200.ops import kernels
from liteinfer_b200.parts import block, side_by_side
from liteinfer_b200.parts.context import AttentionPlan

DEVICE = torch.device("cuda", 0)


class Stream:
    cuda_stream = 0

    def __init__(self) -> None:
        self.waited: list[Stream] = []

    def wait_stream(self, other: "Stream") -> None:
        self.waited.append(other)


@pytest.fixture
def streams(monkeypatch):
    """(the current stream, the second stream) without a GPU."""
    main, second = Stream(), Stream()
    monkeypatch.setattr(kernels.beside, "_streams", {})
    monkeypatch.setattr(kernels.beside, "_open", set())
    monkeypatch.setattr(kernels, "scratch_for", lambda device: None)
    monkeypatch.setattr(torch.cuda, "Stream", lambda device=None: second)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: main)
    monkeypatch.setattr(torch.cuda, "stream", lambda stream: contextlib.nullcontext())
    return main, second


def _fails():
    raise RuntimeError("planted")


def test_an_exception_within_the_lane_joins_it(streams):
    main, second = streams
    lane = ops.beside(DEVICE)
    with pytest.raises(RuntimeError, match="planted"), lane:
        assert not ops.beside.is_free(DEVICE)
        _fails()
    assert main.waited == [second] and ops.beside.is_free(DEVICE)


def test_a_join_that_fails_leaves_the_device_free(streams, monkeypatch):
    main, _ = streams
    with ops.beside(DEVICE) as lane:
        pass
    monkeypatch.setattr(main, "wait_stream", lambda other: _fails())
    with pytest.raises(RuntimeError, match="planted"):
        lane.join()
    assert ops.beside.is_free(DEVICE)


@pytest.mark.parametrize("failing", ["paged_attention_mma", "paged_attention_tcgen05", None])
def test_a_mixed_step_that_fails_joins_its_lane(streams, monkeypatch, failing):
    main, second = streams
    ran = []
    monkeypatch.setattr(kernels, "_on_gpu", lambda *tensors: None)
    monkeypatch.setattr(kernels, "_rows2d", lambda *tensor: None)
    monkeypatch.setattr(kernels, "tcgen05_attention_supports", lambda *sizes: True)
    monkeypatch.setattr(kernels, "stream_attention_supports", lambda *sizes: True)
    for name in ("paged_attention_mma", "paged_attention_tcgen05"):
        monkeypatch.setattr(kernels, name, lambda *a, _name=name, **k: (ran.append((_name, kernels._here.lane)), _name == failing and _fails()))
    ints = lambda *v: torch.tensor(v, dtype=torch.int32)
    q = torch.zeros(5, 64, dtype=torch.bfloat16)
    out = SimpleNamespace(dtype=q.dtype, device=DEVICE)
    pool = torch.zeros(4, 1, 16, 64, dtype=torch.bfloat16)
    plan = AttentionPlan(num_decode=1, decode_seqs=ints(0), decode_tokens=ints(0), num_prefill=1, prefill_seqs=ints(1),
                         max_prefill_query_len=4, max_decode_context_len=9)
    run = lambda: kernels.paged_attention(q, 64, out, pool, pool, torch.zeros(2, 1, dtype=torch.int32), ints(0, 1, 5), ints(9, 4), 2, 4,
                                          1, 1, 64, 0.1, plan=plan)
    if failing is None:
        assert run() is out
        assert ran == [("paged_attention_mma", 1), ("paged_attention_tcgen05", 0)]
    else:
        with pytest.raises(RuntimeError, match="planted"):
            run()
    assert second in main.waited and ops.beside.is_free(DEVICE)


@pytest.mark.parametrize("failing", ["lane", "main"])
def test_a_parallel_layer_that_fails_joins_its_lane(streams, failing):
    main, second = streams
    here = SimpleNamespace(is_cuda=True, shape=(3, 8), device=DEVICE)
    part = lambda fails: SimpleNamespace(gives_sum=True, forward=lambda *args: _fails() if fails else ())
    norm = SimpleNamespace(forward_pair=lambda *args: (None, None))
    layer = block.ParallelNormsBlock({"mixer_norm": norm, "mixer": part(failing == "main"), "feed_forward_norm": norm,
                                      "feed_forward": part(failing == "lane")})
    with pytest.raises(RuntimeError, match="planted"):
        layer.forward(here, None, None, None)
    assert second in main.waited and ops.beside.is_free(DEVICE)


@pytest.mark.parametrize("failing", [0, 1])
def test_mixers_side_by_side_that_fail_join_their_lane(streams, monkeypatch, failing):
    main, second = streams
    monkeypatch.setattr(torch, "empty", lambda *shape, **kw: None)
    monkeypatch.setattr(ops, "linear", lambda *args: None)
    mixers = side_by_side.SideBySide.__new__(side_by_side.SideBySide)
    mixers.members = [SimpleNamespace(mixed_width=8, out_weight=None, mix=lambda *args, _i=i: _i == failing and _fails()) for i in range(2)]
    mixers.in_at, mixers.scales, mixers.out_norms, mixers.norm_eps = [(0, 4), (4, 8)], [1.0, 1.0], [None, None], 1e-5

    class Projection:
        is_cuda, shape, device, dtype = True, (3, 8), DEVICE, torch.bfloat16

        def __getitem__(self, at):
            return self

    with pytest.raises(RuntimeError, match="planted"):
        mixers._normed(Projection(), None, None)
    assert second in main.waited and ops.beside.is_free(DEVICE)


def test_a_thread_does_not_follow_another_to_the_second_stream(streams, monkeypatch):
    """While one thread's launches go to the second stream, another's stay where they were, with the first lane's scratch,
    and the second stream is not to be had."""
    main, second = streams
    second.cuda_stream = 7
    current = threading.local()
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: getattr(current, "stream", main))

    @contextlib.contextmanager
    def on(stream):
        current.stream = stream
        yield
        current.stream = main

    monkeypatch.setattr(torch.cuda, "stream", on)
    seen = []

    def other():
        with kernels.on_current_stream():
            seen.append((kernels._stream(), kernels._here.lane, ops.beside.claim(DEVICE)))

    lane = ops.beside.claim(DEVICE)
    assert ops.beside.claim(DEVICE) is None
    with lane:
        assert (kernels._stream(), kernels._here.lane) == (7, 1)
        thread = threading.Thread(target=other)
        thread.start()
        thread.join()
        assert (kernels._stream(), kernels._here.lane) == (7, 1)
    assert seen == [(0, 0, None)] and (kernels._stream(), kernels._here.lane) == (0, 0)
    lane.join()
    assert ops.beside.claim(DEVICE) is not None


def test_claims_of_many_threads_are_one(streams):
    gate, got = threading.Barrier(8), []

    def run():
        gate.wait()
        got.append(ops.beside.claim(DEVICE))

    threads = [threading.Thread(target=run) for _ in range(8)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert sum(lane is not None for lane in got) == 1
