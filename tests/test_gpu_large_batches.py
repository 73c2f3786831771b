"""Integral and derivative kernels over large batches: a molecule's results do not depend on its batch.

The launch tables hold one entry per molecule and class, which every CTA looks
up; batches sit at the edges of that search (32 entries per step).
"""

import threading

import numpy as np
import pytest
import torch

from vibeqc_b200 import _lib, geometry
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


def _own_plan_gradients(mol, parts, layout):
    """The contractions of one molecule by itself, with its slices of a batch's weights."""
    dens, wdens, mbar, abar = parts
    mat, _, _, met, three = _parts(layout)
    plan = NativePlan([mol], True)
    out = _gradients(plan, dens[mat].clone(), wdens[mat].clone(), mbar[met].clone(), abar[three].clone())
    plan.close()
    return out


def _check_batch(mols, indices):
    plan = NativePlan(mols, True)
    weights = _weights(plan, len(mols))
    got = _gradients(plan, *weights)
    for i in indices:
        lay = plan.layout[i]
        own = _own_plan_gradients(mols[i], weights, lay)
        for g, want in zip(got, own):
            # sums of the same terms in another order: some thousand roundings
            part = g[lay.atom_offset:lay.atom_offset + lay.natom]
            assert (part - want).abs().max().item() <= 1e-12 * (1.0 + want.abs().max().item())
    plan.close()


@pytest.mark.parametrize("count", [1, 32, 33, 1025, 4500])
def test_derivatives_do_not_depend_on_the_batch(count):
    """Molecules of a few chunks: sums straight to global memory."""
    kinds = _molecules()
    step = max(1, count // 23)
    _check_batch([kinds[i % len(kinds)] for i in range(count)],
                 sorted({*range(0, count, step), count - 1}))


@pytest.mark.parametrize("waters,count", [(4, 40), (6, 13)])
def test_shared_sums_over_molecule_boundaries(waters, count):
    """Classes of over 2368 chunks and 96 a molecule: a CTA takes runs of chunks, some across two molecules.

    The runs are 2 to 4 chunks and the molecules' counts no multiples of them
    (114 (ss|s) chunks a (H2O)4, 249 (ss|p)); each molecule has its own
    geometry and weights, so sums added to the neighbour show.
    """
    mols = [make_molecule(geometry.water_cluster(waters, np.random.default_rng([3, i])), "def2-svp",
                          "cc-pvdz-jkfit") for i in range(count)]
    _check_batch(mols, range(0, count, 4))


def _weighted(plan, xyz, dens, wdens, mbar, abar, weight):
    """The three energies whose derivatives the contractions are."""
    f64 = dict(dtype=torch.float64, device="cuda")
    s, t, v = (torch.empty(plan.mat_total, **f64) for _ in range(3))
    m, a = (torch.empty(k, **f64) for k in (plan.met_total, plan.a_total))
    _lib.call("vqc_int1e", plan.handle, xyz.data_ptr(), s.data_ptr(), t.data_ptr(), v.data_ptr(), _stream())
    _lib.call("vqc_int2c", plan.handle, xyz.data_ptr(), m.data_ptr(), _stream())
    _lib.call("vqc_int3c", plan.handle, xyz.data_ptr(), a.data_ptr(), _stream())
    return torch.stack([(dens * (t + v)).sum() - (wdens * s).sum(), (mbar * m).sum(), (weight * abar * a).sum()])


@pytest.mark.parametrize("pairs", [2, 64, 66])  # 4, 128 and 132 atoms: either side of the shared sums' limit
def test_derivatives_against_differences(pairs):
    rng = np.random.default_rng(pairs)
    atoms = [("H", tuple(np.array([3.0 * (i // 2), 0.0, 0.75 * (i % 2)]) + 0.1 * rng.standard_normal(3)))
             for i in range(2 * pairs)]
    plan = NativePlan([make_molecule(atoms, "sto-3g", "cc-pvdz-jkfit")], True)
    lay = plan.layout[0]
    dens, wdens, mbar, abar = _weights(plan, pairs)
    sym = lambda w, k: (w.view(k, k) + w.view(k, k).T).reshape(-1).contiguous()  # noqa: E731
    dens, wdens, mbar = sym(dens, lay.nao), sym(wdens, lay.nao), sym(mbar, lay.naux)
    off = torch.tril_indices(lay.nao, lay.nao, device="cuda")
    weight = torch.where(off[0] == off[1], 1.0, 2.0).double().repeat_interleave(lay.naux)
    grads = _gradients(plan, dens, wdens, mbar, abar)
    x0 = torch.as_tensor(plan.coordinates(), device="cuda").contiguous()
    h = 4e-3
    for atom in (0, pairs, 2 * pairs - 1):
        direction = torch.zeros_like(x0)
        direction[atom] = torch.tensor([0.6, -0.48, 0.64], dtype=torch.float64)
        f = {k: _weighted(plan, (x0 + k * h * direction).contiguous(), dens, wdens, mbar, abar, weight)
             for k in (-2, -1, 1, 2)}
        want = (8 * (f[1] - f[-1]) - (f[2] - f[-2])) / (12 * h)
        for g, w in zip(grads, want):
            # h^4 f'''''/30 with f''''' of the order of (2 a)^2 = 50 f': 5e-10;
            # roundings of sums of up to 3e7 terms over h: below 1e-7
            assert abs(float((g * direction).sum() - w)) < 1e-6 * (1.0 + float(g.abs().max()))
    plan.close()


def _cluster_plan():
    return NativePlan([make_molecule(geometry.water_cluster(3, np.random.default_rng([4, i])), "def2-svp",
                                     "cc-pvdz-jkfit") for i in range(2)], True)


def test_classes_in_order_under_capture():
    """Captured, the classes run in order on one stream: the same results as side by side."""
    plan = _cluster_plan()
    weights = _weights(plan, 5)
    want, want_g = _integrals(plan), _gradients(plan, *weights)
    xyz = torch.as_tensor(plan.coordinates(), device="cuda").contiguous()
    out = [torch.zeros_like(w) for w in want]
    grads = [torch.zeros_like(g) for g in want_g]
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        h, x, st = plan.handle, xyz.data_ptr(), _stream()
        s, t, v, m, a = (o.data_ptr() for o in out)
        _lib.call("vqc_int1e", h, x, s, t, v, st)
        _lib.call("vqc_int2c", h, x, m, st)
        _lib.call("vqc_int3c", h, x, a, st)
        for g in grads:
            g.zero_()
        dens, wdens, mbar, abar = (w.data_ptr() for w in weights)
        _lib.call("vqc_grad1e", h, x, dens, wdens, grads[0].data_ptr(), st)
        _lib.call("vqc_grad2c", h, x, mbar, grads[1].data_ptr(), st)
        _lib.call("vqc_grad3c", h, x, abar, grads[2].data_ptr(), st)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(o, w) for o, w in zip(out, want))
    for g, w in zip(grads, want_g):
        assert (g - w).abs().max().item() <= 1e-12 * (1.0 + w.abs().max().item())
    plan.close()


def test_order_with_the_callers_stream():
    """Inputs written late on the caller's stream, outputs read on it at once."""
    plan = _cluster_plan()
    want = _integrals(plan)
    host = torch.as_tensor(plan.coordinates(), device="cuda").contiguous()
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        xyz = torch.zeros_like(host)
        a = torch.zeros(plan.a_total, dtype=torch.float64, device="cuda")
        torch.cuda._sleep(20_000_000)  # about 10 ms
        xyz.copy_(host)
        _lib.call("vqc_int3c", plan.handle, xyz.data_ptr(), a.data_ptr(), stream.cuda_stream)
        got = a.clone()
        xyz.zero_()  # the next work of the stream must not reach the kernels
        a.zero_()
    stream.synchronize()
    assert torch.equal(got, want[4])
    plan.close()


def test_one_plan_in_two_threads():
    """A call that finds the plan's streams taken runs in order on its own stream."""
    plan = _cluster_plan()
    want = _integrals(plan)
    torch.cuda.synchronize()
    wrong = []

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(50):
                got = _integrals(plan)
                if not all(torch.equal(g, w) for g, w in zip(got, want)):
                    wrong.append(1)
        torch.cuda.synchronize()

    threads = [threading.Thread(target=work) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    plan.close()


def test_full_batches_of_heavy_atoms():
    """512 against 32 molecules of six argon atoms: below six times the time.

    32 leave the GPU half empty; with eight lanes a pair, most without work of
    their own, 512 took eight times as long, with two lanes they take four.
    """
    mol = make_molecule([("Ar", (7.0 * (i % 3), 7.0 * (i // 3), 0.2 * i)) for i in range(6)], "sto-3g", "def2-tzvp")
    times = []
    for count in (32, 512):
        plan = NativePlan([mol] * count, True)
        xyz = torch.as_tensor(plan.coordinates(), device="cuda").contiguous()
        out = [torch.empty(plan.mat_total, dtype=torch.float64, device="cuda") for _ in range(3)]
        times.append(_time(lambda: _lib.call("vqc_int1e", plan.handle, xyz.data_ptr(),
                                             *(o.data_ptr() for o in out), _stream())))
        plan.close()
    assert times[1] < 6 * times[0], times
