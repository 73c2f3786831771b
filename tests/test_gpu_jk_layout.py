"""Layout kernels of the mixed J/K path at the edges of their tiles and vector forms."""

import pytest
import torch

from vibeqc_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,x,ldq,shift", [
    (1, 2, 4, 0), (9, 126, 128, 0), (64, 128, 128, 0), (5000, 116, 116, 0), (17, 130, 136, 0),
    (33, 129, 132, 0), (12, 131, 131, 0), (7, 64, 64, 1)])  # odd x, unpadded rows, unaligned arrays
def test_anchor_combine(rows, x, ldq, shift):
    g = torch.Generator(device="cuda").manual_seed(rows)
    u0 = torch.randn(rows * x + shift, generator=g, device="cuda", dtype=torch.float64)[shift:]
    dh, dl = (scale * torch.randn(rows * ldq + shift, generator=g, device="cuda")[shift:]
              for scale in (1e-2, 1e-6))
    vh, vl = (torch.full((rows * ldq + shift,), 7.0, device="cuda")[shift:] for _ in range(2))
    before = u0.clone()
    st = torch.cuda.current_stream().cuda_stream
    args = (rows, x, ldq)
    _lib.call("vqc_anchor_combine", u0.data_ptr(), dh.data_ptr(), dl.data_ptr(), vh.data_ptr(),
              vl.data_ptr(), *args, 0.5, 0, st)
    assert torch.equal(u0, before)
    du = (dh.double() + dl.double()).view(rows, ldq)[:, :x]
    want = before.view(rows, x) + 0.5 * du
    v = (vh.double() + vl.double()).view(rows, ldq)
    # V is rounded to FP32 (2^-24) and split into two TF32 parts (2^-22 of the value)
    assert ((v[:, :x] - want).abs() <= 2.0**-21 * want.abs()).all()
    assert (vh.view(rows, ldq)[:, x:] == 0).all() and (vl.view(rows, ldq)[:, x:] == 0).all()
    _lib.call("vqc_anchor_combine", u0.data_ptr(), dh.data_ptr(), dl.data_ptr(), 0, 0, *args, 1.0, 1, st)
    # one FP64 product and sum
    bound = 4e-16 * (before.abs().view(rows, x) + du.abs())
    assert ((u0.view(rows, x) - (before.view(rows, x) + du)).abs() <= bound).all()


@pytest.mark.parametrize("nb,n,x,ld", [(1, 1, 1, 4), (2, 24, 116, 24), (1, 31, 33, 32),
                                       (3, 33, 31, 36), (1, 130, 257, 160)])
def test_unpack_aux_major(nb, n, x, ld):
    g = torch.Generator(device="cuda").manual_seed(n)
    bp = torch.randn(nb, n * (n + 1) // 2, x, generator=g, device="cuda", dtype=torch.float64)
    b = torch.full((nb, n, x, ld), 7.0, device="cuda")
    _lib.call("vqc_unpack_aux_major", bp.data_ptr(), nb, n, x, ld, b.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
    i = torch.arange(n, device="cuda")
    hi, lo = torch.maximum(i[:, None], i), torch.minimum(i[:, None], i)
    full = bp[:, hi * (hi + 1) // 2 + lo]  # (nb, mu, nu, Q)
    assert torch.equal(b[..., :n], full.transpose(2, 3).float())
    assert (b[..., n:] == 0).all()


@pytest.mark.parametrize("x,ldq", [(92, 92), (94, 96), (96, 96), (128, 128), (254, 256), (256, 256),
                                   (258, 260), (510, 512)])
def test_anchor_combine_column_groups(x, ldq):
    """Either side of the rule (96 columns) and of the 128-column groups, taken two at a time."""
    test_anchor_combine(300, x, ldq, 0)


@pytest.mark.parametrize("nb,n,x,ld", [(2, 16, 33, 16), (2, 13, 40, 16), (2, 13, 40, 20), (70, 2, 24, 4)])
def test_unpack_aux_major_short_rows(nb, n, x, ld):
    """Either side of the short-row rule (16 columns)."""
    test_unpack_aux_major(nb, n, x, ld)


def _time(call):
    best = float("inf")
    for _ in range(8):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        call()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


def test_rate_of_the_combination_in_place():
    """Mode 1 moves as much as mode 0, so it takes no more than 1.2 of its time (1.26 with one group at a time)."""
    rows, x = 100 * 32 * 20, 500
    u0 = torch.zeros(rows, x, device="cuda", dtype=torch.float64)
    dh, dl, vh, vl = (torch.zeros(rows, x, device="cuda") for _ in range(4))
    st = torch.cuda.current_stream().cuda_stream
    times = [_time(lambda: _lib.call("vqc_anchor_combine", u0.data_ptr(), dh.data_ptr(), dl.data_ptr(),
                                     vh.data_ptr(), vl.data_ptr(), rows, x, x, 1.0, mode, st))
             for mode in (0, 1)]
    assert times[1] < 1.2 * times[0], times


def test_rate_of_short_rows():
    """8192 x (7, 113): 1.5 times a plain conversion of as many elements as are written.

    Tiles of 32 that rows of 8 leave three quarters empty took 2.9 times it.
    """
    nb, n, x, ld = 8192, 7, 113, 8
    bp = torch.zeros(nb, n * (n + 1) // 2, x, device="cuda", dtype=torch.float64)
    b = torch.zeros(nb, n, x, ld, device="cuda")
    src = torch.zeros(b.numel(), device="cuda", dtype=torch.float64)
    st = torch.cuda.current_stream().cuda_stream
    got = _time(lambda: _lib.call("vqc_unpack_aux_major", bp.data_ptr(), nb, n, x, ld, b.data_ptr(), st))
    copy = _time(lambda: b.view(-1).copy_(src))
    assert got < 2.2 * copy, (got, copy)
