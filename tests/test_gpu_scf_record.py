"""The convergence and bookkeeping kernels of an SCF iteration against the elementwise formulas."""

import pytest
import torch

from vibeqc_b200.scf import ANCHOR_COMMUTATOR, DOUBLE_EPS, ENERGY_ROUNDOFF_FACTOR, SCFRecord

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,n,ncol,nspin", [(1, 1, 1, 1), (3, 24, 5, 1), (2, 25, 0, 2), (5, 67, 20, 2),
                                             (2, 300, 50, 1)])
def test_record_matches_elementwise(nb, n, ncol, nspin):
    gen = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda *s: torch.randn(*s, generator=gen, dtype=torch.float64, device="cuda")  # noqa: E731
    ds, cs = [rnd(nb, n, n) for _ in range(nspin)], [rnd(nb, n, ncol) for _ in range(nspin)]
    state = SCFRecord(ds, cs, 1e-10, 1e-8, 1e-8)
    active = torch.ones(nb, dtype=torch.bool, device="cuda")
    e_old = torch.full((nb,), float("nan"), dtype=torch.float64, device="cuda")
    want_it = torch.zeros(nb, dtype=torch.int64, device="cuda")
    f_final = [torch.zeros_like(d) for d in ds]
    d_final, c_final = [d.clone() for d in ds], [c.clone() for c in cs]
    final_de = torch.full_like(e_old, float("inf"))
    final_e, final_drms = torch.zeros_like(e_old), torch.full_like(e_old, float("inf"))
    energy = rnd(nb)
    for it in range(1, 6):
        # from iteration 2 on the first it - 1 molecules meet every criterion; iteration 2 may not
        # end any, so molecule 0 converges in iteration 3, where molecule 1 meets all but the residual
        meets = torch.zeros(nb, dtype=torch.bool, device="cuda")
        if it >= 2:
            meets[: it - 1] = True
        may = it != 2
        new_ds = [torch.where(meets[:, None, None], d + 1e-10 * rnd(nb, n, n), d + rnd(nb, n, n)) for d in ds]
        new_cs, fs = [rnd(nb, n, ncol) for _ in range(nspin)], [rnd(nb, n, n) for _ in range(nspin)]
        energy = torch.where(meets, energy + 1e-12, energy + 1.0)
        cmax = torch.where(meets, torch.full_like(energy, 1e-9), torch.full_like(energy, 1e-4))
        if it == 3 and nb > 2:
            cmax[1] = float("nan")  # never below a tolerance
        de = (energy - e_old).abs().nan_to_num(float("inf"))
        drms = (sum(((a - b) ** 2).sum(dim=(1, 2)) for a, b in zip(new_ds, ds)) / (nspin * n * n)).sqrt()
        guard = ENERGY_ROUNDOFF_FACTOR * DOUBLE_EPS * torch.clamp(
            torch.maximum(energy.abs(), e_old.abs().nan_to_num(0.0)), min=1.0)
        done = (de < 1e-10 + guard) & (drms < 1e-8) & (cmax <= 1e-8) & may
        tight = bool((active & ~(cmax <= ANCHOR_COMMUTATOR)).any())
        keep = active[:, None, None]
        want_it = torch.where(active, torch.full_like(want_it, it), want_it)
        final_de = torch.where(active, de, final_de)
        final_e = torch.where(active, energy, final_e)
        final_drms = torch.where(active, drms, final_drms)
        for s in range(nspin):
            d_final[s] = torch.where(keep, ds[s], d_final[s])
            c_final[s] = torch.where(keep, cs[s], c_final[s])
            f_final[s] = torch.where(keep, fs[s], f_final[s])
        active = active & ~done
        stay = active[:, None, None]
        ds = [torch.where(stay, a, b) for a, b in zip(new_ds, ds)]
        cs = [torch.where(stay, a, b) for a, b in zip(new_cs, cs)]
        e_old = energy
        assert state.step(it, may, energy, cmax, fs, new_ds, new_cs) == (bool(active.any()), tight)
        assert torch.equal(state.active, active) and torch.equal(state.converged, ~active)
        assert torch.equal(state.iterations, want_it) and torch.equal(state.energy_change, final_de)
        assert torch.equal(state.energy, final_e)  # the energy of the last active iteration
        # a sum of at most 2 x 300^2 squares in another order: within 1e-13 of its value
        assert torch.allclose(state.density_rms, final_drms, rtol=1e-13, atol=0.0)
        for got, want in ((state.d, ds), (state.c, cs), (state.d_final, d_final),
                          (state.c_final, c_final), (state.f_final, f_final)):
            assert all(torch.equal(g, w) for g, w in zip(got, want))
        if not bool(active.any()):
            break


@pytest.mark.parametrize("n,nspin", [(1, 1), (24, 1), (67, 2), (300, 2)])
def test_rms_decides_at_the_tolerance(n, nspin):
    """A density change whose rms over all spins lies 1e-6 below or above the tolerance."""
    tol = 1e-8
    f64 = dict(dtype=torch.float64, device="cuda")
    zeros = [torch.zeros(2, n, n, **f64) for _ in range(nspin)]
    factors = [torch.zeros(2, n, 0, **f64) for _ in range(nspin)]
    state = SCFRecord(zeros, factors, 1e-10, tol, tol)
    energy, cmax = torch.full((2,), -5.0, **f64), torch.zeros(2, **f64)
    side = torch.tensor([1.0 - 1e-6, 1.0 + 1e-6], **f64)[:, None, None]
    # the change sits in one spin alone, so a mean over each spin's own size would differ
    change = [torch.full((2, n, n), tol * nspin**0.5, **f64) * side] + [z.clone() for z in zeros[1:]]
    state.step(1, False, energy, cmax, zeros, zeros, factors)  # sets the old energy
    assert state.step(2, True, energy, cmax, zeros, change, factors) == (True, False)
    assert state.converged.tolist() == [True, False] and state.active.tolist() == [False, True]
    assert torch.allclose(state.density_rms, tol * side.flatten(), rtol=1e-12, atol=0.0)
