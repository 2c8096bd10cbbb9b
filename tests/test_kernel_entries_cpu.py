"""The Python side of kernel launches on CPU tensors: the library is a stand-in that writes the same memory through the
raw addresses it is given, so what the wrappers check and record is seen without a GPU."""
import ctypes

import pytest
import torch
import torch.nn.functional as F

from matrix_fsdp_b200.ops import functional as OF
from matrix_fsdp_b200.ops import kernels as K


def _memory(address, shape, dtype):
    n = torch.Size(shape).numel()
    raw = (ctypes.c_char * (n * torch.empty(0, dtype=dtype).element_size())).from_address(address)
    return torch.frombuffer(raw, dtype=dtype).view(shape)


class _Library:
    """What the kernels of the same names do, on host memory."""

    @staticmethod
    def mfsdp_scale(x, is_bf16, n, scale, stream):
        x = _memory(x, (n,), torch.bfloat16 if is_bf16 else torch.float32)
        x.copy_(x.float() * _memory(scale, (1,), torch.float32))
        return 0

    @staticmethod
    def mfsdp_cast_bf16_f32(src, dst, n, stream):
        _memory(dst, (n,), torch.float32).copy_(_memory(src, (n,), torch.bfloat16))
        return 0

    @staticmethod
    def mfsdp_cross_entropy_dev_scale(logits, target, loss, rows, V, ld, scale, ignore_index, stream):
        assert ld == V
        x = _memory(logits, (rows, V), torch.bfloat16)
        xf = x.float().requires_grad_(True)
        with torch.enable_grad():
            want = F.cross_entropy(xf, _memory(target, (rows,), torch.int64), ignore_index=ignore_index, reduction="none")
            (grad,) = torch.autograd.grad(want.sum() * _memory(scale, (1,), torch.float32), xf)
        x.copy_(grad)
        _memory(loss, (rows,), torch.float32).copy_(want.detach())
        return 0


@pytest.fixture
def library(monkeypatch):
    monkeypatch.setattr(K, "_L", lambda: _Library)
    monkeypatch.setattr(K, "_stream", lambda: 0)
    monkeypatch.setattr(OF, "use_native", lambda t: t.dtype == torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_scaling_in_place_is_seen_by_autograd(library, dtype):
    base = torch.randn(24).to(dtype)
    want = (base * 0.5)[8:]
    version = base._version
    assert torch.equal(K.scale_(base[8:], torch.tensor(0.5)), want)
    assert base._version > version


def test_widening_copy_is_seen_by_autograd(library):
    """A graph that saved the destination (a slice of a gradient shard) must not be walked over the new values."""
    src, shard = torch.randn(16).bfloat16(), torch.randn(24)
    w = torch.randn(16, requires_grad=True)
    y = (w * shard[8:]).sum()
    K.cast_bf16_f32(src, shard[8:])
    assert torch.equal(shard[8:], src.float())
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward()


def test_a_scaled_loss_is_not_walked_twice_over_one_graph(library):
    """The logits buffer is used up by the first walk: a second one is refused, as for any saved tensor that was changed
    in place, instead of carrying the factor twice."""
    logits = torch.randn(6, 16).bfloat16().requires_grad_(True)
    target = torch.randint(0, 16, (6,))
    loss = OF.fused_cross_entropy(logits * 1, target) / 2
    (grad,) = torch.autograd.grad(loss, logits, retain_graph=True)
    xf = logits.detach().float().requires_grad_(True)
    (want,) = torch.autograd.grad(F.cross_entropy(xf, target) / 2, xf)
    assert (grad.float() - want).abs().max() <= 2 ** -7 * want.abs().max()      # two bf16 roundings
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(loss, logits)


class _OnDevice(torch.Tensor):
    """A CPU tensor that says it lives on a CUDA device."""

    is_cuda = True

    def get_device(self):
        return 1


@pytest.mark.parametrize("current", [0, 1])
def test_kernels_take_tensors_of_the_current_device_only(library, monkeypatch, current):
    """A launch goes to the current device; tensors of another one keep the torch operations, which switch to it."""
    from matrix_fsdp_b200.ops import lib
    from matrix_fsdp_b200.optim import flat
    from matrix_fsdp_b200.parallel import collectives
    from matrix_fsdp_b200.utils import training

    launched = []
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: current, raising=False)
    monkeypatch.setattr(lib, "available", lambda: True)
    monkeypatch.setattr(flat, "_native", lambda device: True)
    monkeypatch.setattr(K, "sumsq", lambda x: launched.append("sumsq") or x.double().pow(2).sum().float())
    monkeypatch.setattr(K, "scale_", lambda x, s: launched.append("scale") or x.mul_(s))
    monkeypatch.setattr(K, "cast_bf16_f32", lambda s, d: launched.append("cast") or d.copy_(s))

    g = torch.randn(32).as_subclass(_OnDevice)
    before = g.clone()
    training.clip_grad_norm_([], 1.0, extra_grads=[g])
    assert torch.allclose(g.norm(), torch.ones(()), atol=1e-4) and not torch.equal(g, before)

    src, dst = torch.randn(16).bfloat16().as_subclass(_OnDevice), torch.zeros(16).as_subclass(_OnDevice)
    collectives._copy_segment(dst, src)
    assert torch.equal(dst, src.float())

    p, g = torch.randn(16).as_subclass(_OnDevice), torch.randn(16).as_subclass(_OnDevice)
    p.grad = g
    state = dict(exp_avg=torch.zeros(16).as_subclass(_OnDevice), exp_avg_sq=torch.zeros(16).as_subclass(_OnDevice))
    assert flat.FlatShardedAdamW._one_kernel(p, state) == (current == 1)
    assert launched == (["sumsq", "scale", "cast"] if current == 1 else [])
