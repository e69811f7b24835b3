"""The workspace that a step's parts take their buffers from, on the CPU: views kept by size, buffers that move, sizes that creep up."""
import torch

from lia_rs_b200.engine.step import StepRuntime


def cpu_workspace(max_batch_tokens=32):
    runtime = object.__new__(StepRuntime)
    runtime.max_batch_tokens, runtime.device = max_batch_tokens, torch.device("cpu")
    runtime._buffers, runtime._views, runtime.generation = {}, {}, 0
    return runtime


def test_sizes_that_creep_up_move_a_buffer_a_few_times():
    runtime, most = cpu_workspace(), 10000
    for rows in range(1, most // 8 + 1):
        view = runtime.shaped("records", (rows, 8), torch.bfloat16, most)
        assert view.shape == (rows, 8) and view.is_contiguous()
        assert runtime._buffers[("records", torch.bfloat16)].numel() <= max(most, 8 * rows)
    assert runtime.generation <= 12                                     # doublings from 8 to 8192, and the limit
    assert runtime.shaped("records", (most, 8), torch.bfloat16, most).numel() == 8 * most       # beyond it: what is asked for


def test_kept_views_follow_a_buffer_that_moves():
    runtime = cpu_workspace()
    for _ in range(2):                                                  # (a buffer that moves drops all views)
        small, rows = runtime.shaped("a", (4, 4), torch.float32), runtime.workspace("b", (3, 8), torch.float32)
    assert runtime.shaped("a", (4, 4), torch.float32) is small and runtime.workspace("b", (3, 8), torch.float32) is rows
    large = runtime.scratch("a", 1000, torch.float32)
    assert runtime.shaped("a", (4, 4), torch.float32).data_ptr() == large.data_ptr() != small.data_ptr()
    longer = runtime.workspace("b", (40, 8), torch.float32)
    assert runtime.workspace("b", (3, 8), torch.float32).data_ptr() == longer.data_ptr() != rows.data_ptr()


def test_kept_views_are_bounded_and_dropping_them_moves_nothing(monkeypatch):
    monkeypatch.setattr(StepRuntime, "MOST_VIEWS", 5)
    runtime = cpu_workspace()
    at, generation = runtime.scratch("a", 100, torch.float32).data_ptr(), runtime.generation
    for turn in range(2):
        for numel in range(1, 20):
            view = runtime.scratch("a", numel, torch.float32)
            assert view.numel() == numel and view.data_ptr() == at and len(runtime._views) <= 5
    assert runtime.generation == generation


def test_a_shape_may_be_a_list():
    runtime = cpu_workspace()
    view = runtime.workspace("a", [3, 8], torch.float32)
    assert view.shape == (3, 8) and runtime.workspace("a", torch.Size([3, 8]), torch.float32) is view
