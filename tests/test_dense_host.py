"""What ``ops.dense_mm`` hands to its kernel, without a GPU: raw pointers leave Python here, so operands that
are not all on one device, or an output of another shape, have to stop before."""
import contextlib

import pytest
import torch


class _Tensor:
    """What dense_mm asks of a CUDA tensor."""

    is_cuda, dtype = True, torch.float32

    def __init__(self, rows, cols, gpu=0, stride=None, dtype=torch.float32):
        self.shape, self.gpu, self.ld, self.dtype = (rows, cols), gpu, stride or cols, dtype
        self.device = torch.device("cuda", gpu)

    def dim(self):
        return 2

    def stride(self, i):
        return (self.ld, 1)[i]

    def get_device(self):
        return self.gpu

    def data_ptr(self):
        return 256 * (self.gpu + 1)


@pytest.fixture
def world(monkeypatch):
    """A fake library and two fake GPUs; ``calls`` has (current GPU, sizes) of every kernel call."""
    from paramspmm_ae_b200 import ops
    state = dict(current=0, calls=[], mm=0)

    class Lib:
        @staticmethod
        def pspmm_dense_mm(*a):
            state["calls"].append((state["current"], a[2:5]))
            return 0

    @contextlib.contextmanager
    def device(gpu):
        old, state["current"] = state["current"], gpu
        yield
        state["current"] = old

    def mm(a, b):
        state["mm"] += 1
        raise RuntimeError("Expected all tensors to be on the same device")

    monkeypatch.setattr(ops, "lib", lambda: Lib)
    monkeypatch.setattr(ops, "_scratch", lambda *a: (None, 0))
    monkeypatch.setattr(ops, "_stream", lambda: None)
    monkeypatch.setattr(torch, "mm", mm)
    monkeypatch.setattr(torch, "empty", lambda shape, dtype, device: _Tensor(*shape, gpu=device.index))
    monkeypatch.setattr(torch.cuda, "device", device)
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: state["current"], raising=False)
    return ops, state


def test_operands_on_two_gpus_are_an_error(world):
    ops, state = world
    with pytest.raises(RuntimeError, match="same device"):
        ops.dense_mm(_Tensor(4, 8), _Tensor(8, 3, gpu=1))
    assert state["calls"] == [] and state["mm"] == 1


def test_operands_on_another_gpu_are_multiplied_there(world):
    ops, state = world
    out = ops.dense_mm(_Tensor(4, 8, gpu=1), _Tensor(8, 3, gpu=1))
    assert out.gpu == 1 and state["calls"] == [(1, (4, 3, 8))] and state["current"] == 0
    ops.dense_mm(_Tensor(4, 8), _Tensor(8, 3))
    assert state["calls"][1:] == [(0, (4, 3, 8))] and state["mm"] == 0


@pytest.mark.parametrize("out", [dict(rows=4, cols=2), dict(rows=3, cols=3), dict(rows=4, cols=3, gpu=1),
                                 dict(rows=4, cols=3, dtype=torch.float64)])
def test_an_output_that_does_not_fit_is_an_error(world, out):
    ops, state = world
    with pytest.raises(RuntimeError, match="out must be"):
        ops.dense_mm(_Tensor(4, 8), _Tensor(8, 3), out=_Tensor(**out))
    assert state["calls"] == []
    ops.dense_mm(_Tensor(4, 8), _Tensor(8, 3), out=_Tensor(4, 3, stride=7))  # a column slice of a wider array
    assert len(state["calls"]) == 1
