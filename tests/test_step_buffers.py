"""A step's work buffers by name: the same tensor while the shape comes back, one storage a name whatever shapes came before."""
import gc
import weakref

import torch

from mini_engine_b200.engine.step_context import StepContext


class Runner:
    act_dtype, device, error_flag = torch.float32, torch.device("cpu"), None


def test_a_storage_that_grows_leaves_no_earlier_one_behind():
    runner = Runner()
    ctx, seen = StepContext(runner), []
    for rows in (10, 300, 20, 500, 300, 40, 501):
        view = ctx.buffer("states", (rows, 64), torch.float32)
        assert view is ctx.buffer("states", (rows, 64), torch.float32) and view.shape == (rows, 64)
        ctx.buffer("states", (rows,), torch.int32)
        seen.append(weakref.ref(ctx._arena["states"]))
    del view
    gc.collect()
    alive = [s() for s in seen if s() is not None]
    assert {id(s) for s in alive} == {id(ctx._arena["states"])} and alive[0].numel() == 501 * 64 * 4


def test_contexts_that_share_an_arena_follow_a_storage_that_another_replaced():
    runner, arena, replaced = Runner(), {}, []
    one, two = StepContext(runner, arena), StepContext(runner, arena)
    two.on_replace = replaced.append
    small = one.buffer("x", (4,), torch.float32)
    one.buffer("x", (2,), torch.float32)
    old = weakref.ref(arena["x"])
    assert two.buffer("x", (4,), torch.float32).data_ptr() == small.data_ptr() and not replaced
    two.buffer("x", (400,), torch.float32)
    assert replaced == ["x"]
    del small
    assert one.buffer("x", (4,), torch.float32).data_ptr() == arena["x"].data_ptr()
    gc.collect()
    assert old() is None                       # not kept by a view of another shape
    one.frozen = True
    assert one.buffer("x", (4,), torch.float32) is one.buffer("x", (4,), torch.float32)
    try:
        one.buffer("x", (500,), torch.float32)
    except RuntimeError as e:
        assert "captured graph" in str(e)
    else:
        raise AssertionError("a frozen context moved a buffer")


def test_runs_of_a_step_within_the_limits():
    runner = Runner()
    for T, B in ((256, 4), (4096, 64), (100, 512), (16384, 512)):
        runner.max_num_batched_tokens, runner.max_num_seqs = T, B
        most = max(sum(-(-n // 64) for n in lens) for lens in _divisions(T, B))
        assert most <= StepContext(runner).most_runs(64) <= 1.02 * most + 1
        assert StepContext(runner, {}).most_runs(64) == 0


def _divisions(T, B):
    """Steps of T tokens and up to B requests with two tokens and more that are cut into many runs: all but the last just beyond whole runs."""
    for n in range(1, min(B, T // 2) + 1):
        for extra in (2, 65, 129):
            lens = [extra] * (n - 1)
            if sum(lens) + 2 <= T:
                yield lens + [T - sum(lens)]
        k = (T - 2 * n) // 64                 # two tokens each, then whole runs for as many as there are tokens left
        yield [2 + 64 * (k // n + (i < k % n)) for i in range(n)]
