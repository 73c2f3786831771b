"""Integral and derivative kernels over large batches: a molecule's results do not depend on its batch.

The launch tables hold one entry per molecule and class, which every CTA looks
up; batches sit at the edges of that search (32 entries per step).
"""

import numpy as np
import pytest
import torch

from vibeqc_b200 import _lib
from vibeqc_b200.plan import NativePlan, make_molecule

pytestmark = pytest.mark.gpu


def _molecules():
    """Different molecules, so that their classes have different numbers of entries."""
    water = [("O", (0.0, 0.0, 0.1)), ("H", (0.0, 0.76, 0.68)), ("H", (0.1, -0.76, 0.66))]
    atoms = [[("H", (0.0, 0.0, 0.0)), ("H", (0.0, 0.1, 0.74))], [("H", (0.3, 0.0, 0.0)), ("H", (0.0, 0.1, 0.9))],
             water, [("He", (0.1, 0.2, 0.3))]]
    return [make_molecule(a, "def2-svp", "def2-tzvp") for a in atoms]


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _integrals(plan):
    xyz = torch.as_tensor(plan.coordinates(), device="cuda").contiguous()
    f64 = dict(dtype=torch.float64, device="cuda")
    s, t, v = (torch.full((plan.mat_total,), 7.0, **f64) for _ in range(3))
    m, a = (torch.full((k,), 7.0, **f64) for k in (plan.met_total, plan.a_total))
    _lib.call("vqc_int1e", plan.handle, xyz.data_ptr(), s.data_ptr(), t.data_ptr(), v.data_ptr(), _stream())
    _lib.call("vqc_int2c", plan.handle, xyz.data_ptr(), m.data_ptr(), _stream())
    _lib.call("vqc_int3c", plan.handle, xyz.data_ptr(), a.data_ptr(), _stream())
    return s, t, v, m, a


def _weights(plan, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda k: torch.randn(k, generator=g, dtype=torch.float64, device="cuda")  # noqa: E731
    return rnd(plan.mat_total), rnd(plan.mat_total), rnd(plan.met_total), rnd(plan.a_total)


def _gradients(plan, dens, wdens, mbar, abar):
    """The three derivative contractions, (natom, 3) each."""
    xyz = torch.as_tensor(plan.coordinates(), device="cuda").contiguous()
    g1, g2, g3 = (torch.zeros(plan.natom, 3, dtype=torch.float64, device="cuda") for _ in range(3))
    h, x, st = plan.handle, xyz.data_ptr(), _stream()
    _lib.call("vqc_grad1e", h, x, dens.data_ptr(), wdens.data_ptr(), g1.data_ptr(), st)
    _lib.call("vqc_grad2c", h, x, mbar.data_ptr(), g2.data_ptr(), st)
    _lib.call("vqc_grad3c", h, x, abar.data_ptr(), g3.data_ptr(), st)
    return g1, g2, g3


def _parts(layout):
    """Slices of a molecule's blocks in (s, t, v, metric, three-centre) arrays."""
    mat = slice(layout.mat_offset, layout.mat_offset + layout.nao ** 2)
    met = slice(layout.met_offset, layout.met_offset + layout.naux ** 2)
    three = slice(layout.a_offset, layout.a_offset + layout.npair * layout.naux)
    return mat, mat, mat, met, three


@pytest.mark.parametrize("count", [1, 31, 32, 33, 64, 1023, 1025, 4500])
def test_integrals_do_not_depend_on_the_batch(count):
    kinds = _molecules()
    singles = []
    for mol in kinds:
        plan = NativePlan([mol], True)
        singles.append(_integrals(plan))
        plan.close()
    plan = NativePlan([kinds[i % len(kinds)] for i in range(count)], True)
    got = _integrals(plan)
    step = max(1, count // 61)
    for i in sorted({*range(0, count, step), max(0, count - 2), count - 1}):
        for arr, sl, want in zip(got, _parts(plan.layout[i]), singles[i % len(kinds)]):
            # the order of sums may depend on the launch: a few roundings of values below 100
            assert (arr[sl] - want).abs().max().item() < 1e-12
    plan.close()


def _time(call):
    best = float("inf")
    for _ in range(6):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        call()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


def test_cost_of_small_molecules():
    """One-electron kernels over H2: the look-up does not grow with the batch, no CTA is empty.

    Eight times the molecules may take sixteen times the time (a look-up linear
    in the number of molecules made it above 60).  The 3 pairs of a molecule
    with 2 nuclei are less work than its 3-centre integrals: with seven of eight
    CTAs empty they took 0.8 of that time, without 0.2.
    """
    mol = make_molecule([("H", (0.0, 0.0, 0.0)), ("H", (0.0, 0.0, 0.74))], "sto-3g", "cc-pvdz-jkfit")
    times = []
    for count in (4096, 32768):
        plan = NativePlan([mol] * count, True)
        xyz = torch.as_tensor(plan.coordinates(), device="cuda").contiguous()
        out = [torch.empty(plan.mat_total, dtype=torch.float64, device="cuda") for _ in range(3)]
        times.append(_time(lambda: _lib.call("vqc_int1e", plan.handle, xyz.data_ptr(),
                                             *(o.data_ptr() for o in out), _stream())))
    a = torch.empty(plan.a_total, dtype=torch.float64, device="cuda")
    three = _time(lambda: _lib.call("vqc_int3c", plan.handle, xyz.data_ptr(), a.data_ptr(), _stream()))
    assert times[1] < 16 * times[0], times
    assert times[1] < 0.5 * three, (times, three)
