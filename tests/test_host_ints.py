"""Host integers that reach the device as launch arguments (``ops.ints_on``, ``ops.set_ints``)."""
import ctypes
import threading

import pytest
import torch

from trimkv_b200 import _lib, ops


def test_argument_errors_without_a_gpu():
    lib, one, seen = _lib.lib(), 16, []

    def calls():                         # the error text is one per thread: the main thread's stays as it is
        seen.append(lib.tkv_put_ints(None, None, 0, None) == 0 and lib.tkv_set_ints(None, None, 0, 0, None) == 0)
        seen.append(lib.tkv_put_ints(one, None, 3, None) == -1 and lib.tkv_put_ints(None, None, -1, None) == -1)
        seen.append(lib.tkv_set_ints(one, None, 3, 0, None) == -1)
        seen.append(lib.tkv_set_ints(one, (ctypes.c_int32 * 2)(4, -1), 2, 0, None) == -1 and b"index -1" in lib.tkv_last_error())
    t = threading.Thread(target=calls)
    t.start()
    t.join()
    assert seen == [True] * 4


def test_host_tensors():
    assert ops.ints_on(torch.device("cpu"), [3, 1, 2]).tolist() == [3, 1, 2]
    t = torch.arange(5, dtype=torch.int32)
    ops.set_ints(t, [4, 1], 9)
    assert t.tolist() == [0, 9, 2, 3, 9]


# argument blocks of 60 and of 960 integers, and more than one launch
@pytest.mark.gpu
@pytest.mark.parametrize("n", [0, 1, 59, 60, 61, 959, 960, 961, 2500])
def test_values_arrive(n):
    dev = torch.device("cuda", 0)
    g = torch.Generator().manual_seed(n)
    values = torch.randint(-2 ** 31, 2 ** 31 - 1, (n,), generator=g).tolist()
    got = ops.ints_on(dev, values)
    assert got.dtype == torch.int32 and got.tolist() == values
    t = torch.arange(4000, dtype=torch.int32, device=dev)
    index = torch.randperm(4000, generator=g)[:n].tolist()
    ops.set_ints(t, index, -7)
    want = torch.arange(4000, dtype=torch.int32)
    want[index] = -7
    assert torch.equal(t.cpu(), want)
    with pytest.raises(IndexError):
        ops.set_ints(t, [4000], 0)


@pytest.mark.gpu
def test_refused_while_capturing():
    dev = torch.device("cuda", 0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        with pytest.raises(RuntimeError, match="captured"):
            ops.ints_on(dev, [1])
    graph.reset()


def test_takes_what_a_tensor_takes():
    """``want`` of a packed forward pass may hold whatever an int32 tensor is made of; beyond 32 bits is an error, not another row."""
    np = pytest.importorskip("numpy")
    cpu = torch.device("cpu")
    assert ops.ints_on(cpu, [torch.tensor(5), np.int64(7), True, 2.0]).tolist() == [5, 7, 1, 2]
    t = torch.zeros(4, dtype=torch.int32)
    for far in (2 ** 31, -2 ** 31 - 1, 2 ** 32 + 1):
        with pytest.raises(RuntimeError, match="overflow"):
            ops.ints_on(cpu, [0, far])
        with pytest.raises(RuntimeError, match="overflow"):
            ops.set_ints(t, [1], far)
        with pytest.raises(IndexError):
            ops.set_ints(t, [far], 0)
    with pytest.raises(IndexError):
        ops.set_ints(t, [4], 0)
    with torch.device("meta"):                   # a default device of another kind changes nothing
        assert ops.ints_on(cpu, [1]).device == cpu


@pytest.mark.gpu
def test_takes_what_a_tensor_takes_on_the_gpu():
    np = pytest.importorskip("numpy")
    dev = torch.device("cuda", 0)
    mixed = [torch.tensor(5), torch.tensor(6, device=dev), np.int64(7), True, 2.0]
    assert ops.ints_on(dev, mixed).tolist() == [5, 6, 7, 1, 2]
    with pytest.raises(RuntimeError, match="overflow"):
        ops.ints_on(dev, [2 ** 32 + 1])
    with pytest.raises(RuntimeError, match="overflow"):
        ops.set_ints(torch.zeros(4, dtype=torch.int32, device=dev), [1], 2 ** 32 + 1)
