"""decode_matmul_sequence hands raw addresses to the library, so everything that makes them valid is checked before:
on the CPU, with tensors that pass for CUDA ones and a library that only records its arguments."""
import contextlib
import ctypes
import gc
import types
import weakref

import pytest
import torch

from decode_matmul_b200 import _lib, ops


class Dev(torch.Tensor):
    """A CPU tensor that says it lives on CUDA device ``index``."""
    index = 0
    is_cuda = True

    def get_device(self):
        return self.index

    @property
    def device(self):
        return torch.device("cuda", self.index)


def dev(shape, dtype, index=0):
    t = torch.zeros(shape, dtype=dtype).as_subclass(Dev)
    t.index = index
    return t


def layer(n, k, index=0, codebook=(256, 8)):
    return types.SimpleNamespace(codes=dev((n, k // 8), torch.int16, index), codebook=dev(codebook, torch.float16, index), scale=0.5)


@pytest.fixture
def calls(monkeypatch):
    """Argument tuples that reached the library."""
    seen = []

    class Fake:
        def dmm_f16_sequence(self, arr, n, M, *rest):
            seen.append(([(arr[i].x, arr[i].codes, arr[i].out, arr[i].N, arr[i].K, arr[i].zero_ptr) for i in range(n)], M, rest))
            return 0

    fake = Fake()
    monkeypatch.setattr(ops._lib, "lib", lambda: fake)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 0)
    return seen


def test_addresses_arrive_in_order(calls):
    x, a, g = dev((3, 64), torch.float32), dev((3, 32), torch.float32), dev((7,), torch.float32)
    first, second, nxt = layer(32, 64), layer(64, 32), layer(48, 32)
    block = [ops.fused_op(x, first, a, zero=g), ops.fused_op(a, second, x)]
    ops.decode_matmul_sequence(block, 3, x.device, next_weights=nxt, workspace=dev((256,), torch.uint8))
    (got, M, rest), = calls
    assert M == 3 and rest[2:5] == (nxt.codes.data_ptr(), 48, 32) and rest[6] == 256
    assert got == [(x.data_ptr(), first.codes.data_ptr(), a.data_ptr(), 32, 64, g.data_ptr()),
                   (a.data_ptr(), second.codes.data_ptr(), x.data_ptr(), 64, 32, None)]


@pytest.mark.parametrize("M", [2, 4, 64])
def test_every_op_has_m_rows(calls, M):
    ok = ops.fused_op(dev((M, 64), torch.float32), layer(32, 64), dev((M, 32), torch.float32))
    bad = ops.fused_op(dev((3, 64), torch.float32), layer(32, 64), dev((3, 32), torch.float32))
    for block in ([bad], [ok, bad], [bad, ok]):
        with pytest.raises(RuntimeError, match="rows"):
            ops.decode_matmul_sequence(block, M, "cuda")
    assert not calls


def test_everything_is_on_one_device(calls):
    x, out = dev((1, 64), torch.float32), dev((1, 32), torch.float32)
    for lin, o, z in ((layer(32, 64, 1), out, None), (layer(32, 64), dev((1, 32), torch.float32, 1), None),
                      (layer(32, 64), out, dev((8,), torch.float32, 1))):
        with pytest.raises(RuntimeError, match="device"):
            ops.fused_op(x, lin, o, zero=z)
    here = ops.fused_op(x, layer(32, 64), out)
    there = ops.fused_op(dev((1, 64), torch.float32, 1), layer(32, 64, 1), dev((1, 32), torch.float32, 1))
    for args, kw in ((([here, there], 1, "cuda"), {}), (([there], 1, "cuda"), {}), (([here], 1, "cuda:1"), {}),
                     (([here], 1, "cuda"), {"next_weights": layer(32, 64, 1)}),
                     (([here], 1, "cuda"), {"workspace": dev((256,), torch.uint8, 1)})):
        with pytest.raises(RuntimeError, match="device"):
            ops.decode_matmul_sequence(*args, **kw)
    assert not calls


def test_operands_are_what_the_kernels_read():
    x, out = dev((1, 64), torch.float32), dev((1, 32), torch.float32)
    with pytest.raises(RuntimeError, match="codebook"):
        ops.fused_op(x, layer(32, 64, codebook=(128, 8)), out)
    with pytest.raises(RuntimeError, match="CUDA"):
        ops.fused_op(torch.zeros((1, 64)), layer(32, 64), out)
    with pytest.raises(RuntimeError, match="contiguous"):
        ops.fused_op(dev((64, 1), torch.float32).t()[:, ::2], layer(32, 32), out)
    with pytest.raises(RuntimeError, match="dtype"):
        ops.fused_op(x.double(), layer(32, 64), out)


def test_an_op_keeps_its_tensors():
    """The tensors of an op live until the op does: their memory must not be given out again before the launch."""
    lin = layer(32, 64)
    refs, made = [], []
    for shape in ((1, 64), (1, 32), (8,)):
        made.append(dev(shape, torch.float32))
        refs.append(weakref.ref(made[-1]))
    op = ops.fused_op(made[0], lin, made[1], zero=made[2])
    del made
    gc.collect()
    assert all(r() is not None for r in refs)
    del op
    gc.collect()
    assert all(r() is None for r in refs)


def test_status_codes_of_the_c_entry():
    """Null, no ops, and a first op that is refused: codes, before anything is launched."""
    L = _lib.lib()
    assert L.dmm_f16_sequence(None, 1, 1, 0, 0, None, 0, 0, None, 0, None) == -1
    arr = (_lib.FusedOp * 2)()
    assert L.dmm_f16_sequence(arr, 0, 1, 0, 0, None, 0, 0, None, 0, None) == -4
    assert L.dmm_f16_sequence(arr, 1, 1, 0, 0, None, 0, 0, None, 0, None) == -1  # null operands
    buf = (ctypes.c_char * 4096)()
    p = (ctypes.addressof(buf) + 255) & ~255
    bad = _lib.FusedOp(p, _lib.X_F32, 32, 0, p, p, 1.0, p, 24, 32, None, 0)
    assert L.dmm_f16_sequence((_lib.FusedOp * 1)(bad), 1, 1, 0, 0, None, 0, 0, None, 0, None) == -2
    assert L.dmm_f16_sequence((_lib.FusedOp * 1)(bad), 1, 1, 0, 0, p, 24, 32, None, 0, None) == -2  # the matrix that follows
