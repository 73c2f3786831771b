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
    energy = rnd(nb)
    for it in range(1, 6):
        # molecule it - 2 meets every criterion in iteration it >= 2 but the third only in phase 4+
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
        for got, want in ((state.d, ds), (state.c, cs), (state.d_final, d_final),
                          (state.c_final, c_final), (state.f_final, f_final)):
            assert all(torch.equal(g, w) for g, w in zip(got, want))
        if not bool(active.any()):
            break
