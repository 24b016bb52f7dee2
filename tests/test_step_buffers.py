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
