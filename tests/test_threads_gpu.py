"""Two threads that step engines of their own at the same time."""

from __future__ import annotations

import threading

import pytest
import torch

import tiny_configs

pytestmark = pytest.mark.gpu


def _steps(runner, vocab: int, seed: int) -> list[torch.Tensor]:
    """Mixed steps: a request decodes beside portions of another's prompt, over and over."""
    from liteinfer_b200.engine.runner import StepEntry

    g = torch.Generator().manual_seed(seed)
    draw = lambda n: torch.randint(0, vocab, (n,), generator=g).tolist()
    out = [runner.step([StepEntry("a", draw(70), (69,))]).clone()]
    for i in range(12):
        n = int(torch.randint(2, 60, (1,), generator=g))
        out.append(runner.step([StepEntry("a", draw(1), (0,)), StepEntry(f"p{i}", draw(n), (n - 1,))]).clone())
        out.append(runner.step([StepEntry("a", draw(1), (0,)), StepEntry(f"p{i}", draw(3), (0, 2))]).clone())
        runner.release(f"p{i}")
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("name", ["tiny_d", "tiny_e"])
def test_two_threads_step_side_by_side(model_dirs, name):
    """Each thread's mixed steps give what they give alone: neither follows the other to the second stream."""
    from liteinfer_b200 import ops
    from liteinfer_b200.engine.loading import build_runner

    config, _, page = tiny_configs.ALL[name]
    make = lambda: build_runner(model_dirs[name], torch.bfloat16, "cuda:0", page, 64, 4)
    alone = [_steps(make(), config["vocab_size"], seed) for seed in (1, 2)]
    runners, got, gate = [make(), make()], [None, None], threading.Barrier(2)

    def run(i: int) -> None:
        gate.wait()
        got[i] = _steps(runners[i], config["vocab_size"], i + 1)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    for mine, theirs in zip(alone, got):
        assert theirs is not None and all(torch.equal(a, b) for a, b in zip(mine, theirs, strict=True))
    assert ops.beside.is_free(torch.device("cuda:0")) and ops.gemm_error_flag("cuda:0") == 0
