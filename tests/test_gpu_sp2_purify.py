"""One-launch FP64 purification against eigenvectors, over the forms' edges.

Sizes sit at the edges of the 8-, 16-, 32- and 64-row tiles, of the 32-column
K stages and of the one-CTA form; batches at one molecule, several groups and
more molecules than resident groups.
"""

import threading

import pytest
import torch

from vibeqc_b200 import _lib
from vibeqc_b200.scf import _purify_fp64, purify_sp2

pytestmark = pytest.mark.gpu


def _fock(nb, n, nocc, seed):
    """Symmetric matrices with a gap of 0.6 in a spectrum of width about 25, as a Fock matrix has."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = dict(generator=g, dtype=torch.float64, device="cuda")
    q = torch.linalg.qr(torch.randn(nb, n, n, **rnd))[0]
    lam = torch.cat([-0.5 - 20.0 * torch.rand(nb, nocc, **rnd) ** 3,
                     0.1 + 4.0 * torch.rand(nb, n - nocc, **rnd)], dim=1)
    f = (q * lam[:, None, :]) @ q.transpose(1, 2)
    v = q[:, :, :nocc]
    return 0.5 * (f + f.transpose(1, 2)), v @ v.transpose(1, 2)


@pytest.mark.parametrize("path,nb,n", [
    (1, 1, 2), (1, 3, 7), (1, 2, 8), (1, 5, 17), (1, 200, 24), (1, 2, 64), (1, 2, 105), (1, 1, 112),
    (2, 1, 2), (2, 1, 31), (2, 3, 33), (2, 2, 65), (2, 1, 96), (2, 700, 40), (2, 2, 257),
    (3, 1, 5), (3, 1, 64), (3, 2, 63), (3, 3, 129), (3, 400, 70), (3, 2, 384), (0, 2, 64), (0, 2, 66),
    (0, 1, 700)])
def test_projector_matches_eigenvectors(path, nb, n):
    nocc = max(1, n // 5)
    f, want = _fock(nb, n, nocc, 100 * n + nb)
    got = _purify_fp64(f, nocc, 96, 1e-11, path)
    # two steps past tr X - tr X^2 < 1e-11 X is idempotent, and it commutes with F, to rounding:
    # eigenvector error <= n eps |F| / gap = 700 * 2.2e-16 * 25 / 0.6 < 7e-12
    assert (got - want).abs().max().item() < 2e-11
    assert torch.equal(got, got.transpose(1, 2))


@pytest.mark.parametrize("path,n", [(1, 30), (2, 80), (3, 80)])
def test_step_cap_and_occupations(path, n):
    f, _ = _fock(2, n, 4, n)
    # no step: X is the mapped matrix, whose eigenvalues lie in [0, 1]
    x0 = torch.linalg.eigvalsh(_purify_fp64(f, 4, 0, 1e-11, path))
    assert x0.min().item() > -1e-12 and x0.max().item() < 1 + 1e-12
    # nothing occupied, everything occupied
    assert _purify_fp64(f, 0, 96, 1e-11, path).abs().max().item() < 1e-11
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    assert (_purify_fp64(f, n, 96, 1e-11, path) - eye).abs().max().item() < 1e-11
    # non-finite input stays visible and leaves the neighbours alone
    bad = f.clone()
    bad[1, 3, 5] = float("nan")
    got = _purify_fp64(bad, 4, 96, 1e-11, path)
    assert torch.isnan(got[1]).any() and torch.equal(got[0], _purify_fp64(f[:1], 4, 96, 1e-11, path)[0])


def test_layouts_and_arguments():
    f, want = _fock(3, 48, 9, 1)
    strided = f.repeat_interleave(2, dim=2)[:, :, ::2]
    assert (purify_sp2(strided, 9) - want).abs().max().item() < 2e-11
    with pytest.raises(_lib.VqcError):
        _purify_fp64(_fock(1, 113, 9, 1)[0], 9, 96, 1e-11, 1)


@pytest.mark.parametrize("path,nb,n", [(2, 1, 512), (0, 1, 1000), (3, 1, 1400), (0, 2, 700)])
def test_groups_of_many_tiles(path, nb, n):
    """More tiles than the 128 CTAs a group once had, up to every resident CTA."""
    f, want = _fock(nb, n, n // 5, n)
    got = _purify_fp64(f, n // 5, 96, 1e-11, path)
    assert (got - want).abs().max().item() < 4e-11  # n eps |F| / gap, as above, at n = 1400
    assert torch.equal(got, got.transpose(1, 2))


@pytest.mark.parametrize("n", [512, 1000])
def test_one_large_molecule_uses_every_cta(n):
    """About 50 squarings with their updates: less than the time of 85 library squarings.

    Groups of at most 128 CTAs took 108 (n = 512) and 99 (n = 1000) of them, every CTA 62 and 39.
    """
    f, _ = _fock(1, n, n // 5, n)
    times = []
    for call in (lambda: _purify_fp64(f, n // 5, 96, 1e-11),
                 lambda: [torch.bmm(f, f) for _ in range(85)]):
        best = float("inf")
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            call()
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    assert times[0] < times[1], times


@pytest.mark.parametrize("path", [0, 1, 2, 3])
def test_bounds_that_are_eigenvalues(path):
    """One function, multiples of the identity and diagonal matrices: the map has no room beside the spectrum."""
    f64 = dict(dtype=torch.float64, device="cuda")
    for n in (1, 5, 70):
        eye = torch.eye(n, **f64).expand(3, n, n)
        for f in (-0.9 * eye, torch.zeros(3, n, n, **f64), torch.diag(torch.linspace(-2.0, 1.0, n, **f64)).expand(3, n, n)):
            f = f.contiguous()
            assert torch.equal(_purify_fp64(f, n, 96, 1e-11, path), eye)
            assert torch.equal(_purify_fp64(f, 0, 96, 1e-11, path), torch.zeros_like(f))
        bad = f.clone()
        bad[1, 0, n - 1] = float("nan")
        got = _purify_fp64(bad, n, 96, 1e-11, path)
        assert torch.isnan(got[1, 0, n - 1]) and torch.equal(got[0], eye[0]) and torch.equal(got[2], eye[2])
    # one of two degenerate levels: no projector, and none is made up
    assert torch.isnan(_purify_fp64(torch.eye(2, **f64)[None].contiguous(), 1, 96, 1e-11, path)).any()
    f = torch.diag(torch.tensor([-2.0, -1.0, 0.5, 1.0], **f64))[None].contiguous()
    want = torch.diag(torch.tensor([1.0, 1.0, 0.0, 0.0], **f64))[None]
    assert (_purify_fp64(f, 2, 96, 1e-11, path) - want).abs().max().item() < 1e-12


@pytest.mark.parametrize("gemm", ["fp64", "int8"])
def test_everything_occupied_in_either_form(gemm):
    f = torch.diag(torch.tensor([-2.0, -1.0, -1.0], dtype=torch.float64, device="cuda"))[None].contiguous()
    eye = torch.eye(3, dtype=torch.float64, device="cuda")[None]
    assert torch.equal(purify_sp2(f, 3, gemm=gemm), eye)
    assert torch.equal(purify_sp2(f, 0, gemm=gemm), torch.zeros_like(f))


@pytest.mark.parametrize("nb,n", [(4, 264), (1, 512), (40, 64)])
def test_two_threads_at_once(nb, n):
    """Each launch brings its own workspace, and a cooperative launch is resident as a whole."""
    f, _ = _fock(nb, n, n // 5, n)
    want = _purify_fp64(f, n // 5, 96, 1e-11)
    torch.cuda.synchronize()
    wrong = []

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(10):
                if not torch.equal(_purify_fp64(f, n // 5, 96, 1e-11), want):
                    wrong.append(1)

    threads = [threading.Thread(target=work) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
