"""The neighbour list at the ends of its index range."""
import ctypes

import numpy as np
import pytest

from fourierd3_b200 import _native


def test_a_count_beyond_the_row_starts_is_refused():
    # refused on the host, before the pointers (never read here) reach a launch
    lib = _native.lib()
    cell, size = np.eye(3).reshape(9) * 20.0, ctypes.c_size_t()
    _native.check(lib.fd3_neighbor_workspace_size(10, _native.dptr(cell), 6.0, ctypes.byref(size)), "size")
    p = ctypes.c_void_p(256)
    for count in (-1, 2**31, 2**40):
        assert lib.fd3_neighbor_fill_counted(10, p, _native.dptr(cell), 6.0, p, size.value, count, p, p, p,
                                             None) == _native.FD3_EINVAL


def test_the_counted_fill_checks_its_arguments_on_the_host():
    # no list to build: nothing is launched, and outputs may be absent; each bad argument by itself is refused
    lib = _native.lib()
    cell, size, p = np.eye(3).reshape(9) * 20.0, ctypes.c_size_t(), ctypes.c_void_p(256)
    _native.check(lib.fd3_neighbor_workspace_size(10, _native.dptr(cell), 6.0, ctypes.byref(size)), "size")

    def fill(n=10, pos=p, h=_native.dptr(cell), r=6.0, work=p, room=size.value, count=5, src=p, dst=p, shift=p):
        return lib.fd3_neighbor_fill_counted(n, pos, h, r, work, room, count, src, dst, shift, None)

    assert fill(count=0, src=None, dst=None, shift=None) == _native.FD3_OK
    for bad in (dict(n=0), dict(n=2**30 + 1), dict(pos=None), dict(h=None), dict(r=0.0), dict(src=None), dict(dst=None),
                dict(shift=None), dict(h=_native.dptr(np.zeros(9)))):
        assert fill(**bad) == _native.FD3_EINVAL, bad
    assert fill(work=None) == fill(room=size.value - 1) == _native.FD3_ENOMEM


@pytest.mark.gpu
def test_more_pairs_than_the_row_starts_hold_are_refused_with_their_number(cuda_device):
    # 66,000 atoms with about half of all others and their images in reach: 2.28e9 pairs
    import torch

    lib = _native.lib()
    n, cell = 66000, np.eye(3).reshape(9) * 12.1
    pos = torch.rand((n, 3), dtype=torch.float64, device=cuda_device, generator=torch.Generator(cuda_device).manual_seed(1)) * 12.1
    size, count = ctypes.c_size_t(), ctypes.c_int64()
    _native.check(lib.fd3_neighbor_workspace_size(n, _native.dptr(cell), 6.0, ctypes.byref(size)), "size")
    work = torch.empty(size.value, dtype=torch.uint8, device=cuda_device)
    rc = lib.fd3_neighbor_count(n, pos.data_ptr(), _native.dptr(cell), 6.0, work.data_ptr(), size.value,
                                ctypes.byref(count), torch.cuda.current_stream().cuda_stream)
    assert rc == _native.FD3_ECAPACITY
    # pairs of uniform points: n (n - 1) times the sphere's share of the cell, to its statistical error
    want = n * (n - 1) * 4.0 / 3.0 * np.pi * 6.0**3 / 12.1**3
    assert count.value > 2**31 and abs(count.value - want) <= 1e-3 * want


@pytest.mark.gpu
@pytest.mark.parametrize("room", [0, 1, 997])
def test_the_counted_fill_stays_within_the_count_it_is_given(cuda_device, room):
    # fewer pairs than were counted: the first ones are written, the space behind them is untouched
    import torch

    from fourierd3_b200 import neighbour_list

    lib = _native.lib()
    n, cell = 300, np.eye(3).reshape(9) * 13.0
    pos = torch.rand((n, 3), dtype=torch.float64, device=cuda_device, generator=torch.Generator(cuda_device).manual_seed(2)) * 13.0
    i, j, s = neighbour_list(pos, cell.reshape(3, 3), 6.0)
    size, count = ctypes.c_size_t(), ctypes.c_int64()
    _native.check(lib.fd3_neighbor_workspace_size(n, _native.dptr(cell), 6.0, ctypes.byref(size)), "size")
    work = torch.empty(size.value, dtype=torch.uint8, device=cuda_device)
    stream = torch.cuda.current_stream().cuda_stream
    args = (n, pos.data_ptr(), _native.dptr(cell), 6.0, work.data_ptr(), size.value)
    _native.check(lib.fd3_neighbor_count(*args, ctypes.byref(count), stream), "count")
    m = count.value
    src, dst = (torch.full((m,), -7, dtype=torch.int64, device=cuda_device) for _ in range(2))
    shift = torch.full((m, 3), -7, dtype=torch.int32, device=cuda_device)
    _native.check(lib.fd3_neighbor_fill_counted(*args, room, src.data_ptr(), dst.data_ptr(), shift.data_ptr(), stream),
                  "fill")
    for got, want in ((src, i), (dst, j), (shift, s)):
        assert torch.equal(got[:room], want[:room]) and bool((got[room:] == -7).all())
