"""Timed cases: the work a program has this engine do, through its entry points.

A case names one entry point (``kind``) and the sizes of its call.  Whole calls
(``singlepoint``, ``execute``, ``autograd``, ``uhf``, ``fock``) run as a program
runs them, host coordinates or densities in and energies, forces and matrices
out; the others are the layers a program that drives the pieces itself calls
(integrals, whitening, J/K builds, purification, derivative contraction), each
on one homogeneous group of molecules resident on the device.

Molecules are the repository's synthetic ones: water clusters of 1 to 16
molecules (24 to 384 basis functions in def2-SVP, cc-pVDZ-JKFIT auxiliary) and
short alkanes, with geometries made from the seed.  SCF runs start from the
core-Hamiltonian guess (no warm start), so every pass does the same work.
"""

import numpy as np
import torch

from vibeqc_b200 import Calculator, FockPlan, _lib, geometry
from vibeqc_b200 import jk as jkmod
from vibeqc_b200 import scf
from vibeqc_b200.basis import atomic_number
from vibeqc_b200.plan import NativePlan, make_molecule
from vibeqc_b200.torch import batched_energy

BASIS, AUX = "def2-svp", "cc-pvdz-jkfit"
AUX_CARBON = "def2-tzvp"  # no carbon JK-fit set is bundled


def listed():
    return [
        # one molecule at a time with the default options (FP64): the first
        # call of every user, bound by launches and host work
        {"name": "singlepoint_water", "kind": "singlepoint", "waters": 1},
        # the ragged production batch of the benchmark, cut to about 1 s:
        # every size of 2..16 waters, energies and forces, mixed precision
        {"name": "execute_clusters_mixed", "kind": "execute", "count": 30, "n_min": 2, "n_max": 16,
         "precision": "mixed"},
        # training a force model on molecules: batched energies and their
        # autograd gradients with device coordinates, FP64
        {"name": "autograd_alkanes", "kind": "autograd", "count": 8, "n_min": 2, "n_max": 5},
        # open shells: doublet cations of water clusters, energies and forces
        {"name": "uhf_cations_mixed", "kind": "uhf", "count": 12, "n_min": 1, "n_max": 6,
         "precision": "mixed"},
        # J/K source of a hybrid-DFT program: one cluster, a new density in,
        # Fock matrices and the two-electron gradient out
        {"name": "fock_plan_h2o7", "kind": "fock", "waters": 7},
        # integrals of a new geometry: 1-electron, metric and 3-centre tensor
        {"name": "integrals_h2o9x8", "kind": "integrals", "waters": 9, "count": 8},
        # derivative-integral contraction with given weights (the backward direction)
        {"name": "gradient_h2o6x12", "kind": "gradient", "waters": 6, "count": 12},
        # whitening B = A W of the 3-centre tensor, once per geometry
        {"name": "whiten_h2o10x8", "kind": "whiten", "waters": 10, "count": 8},
        # density purification of every SCF iteration
        {"name": "purify_h2o13x14", "kind": "purify", "waters": 13, "count": 14},
        # mixed J/K build of an SCF iteration: many small molecules
        {"name": "jk_h2o3x32", "kind": "jk", "waters": 3, "count": 32},
        # the same for the largest clusters
        {"name": "jk_h2o16x8", "kind": "jk", "waters": 16, "count": 8},
        # increment about the FP64 anchor: the iterations near convergence
        {"name": "jk_increment_h2o11x10", "kind": "jk_increment", "waters": 11, "count": 10},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["singlepoint", "execute", "autograd", "uhf", "fock", "integrals", "gradient",
                       "whiten", "purify", "jk", "jk", "jk_increment"])
    if kind == "singlepoint":
        return {"kind": kind, "waters": rng.randint(2, 6)}
    if kind == "execute":
        lo = rng.randint(1, 9)
        return {"kind": kind, "count": rng.randint(2, 20), "n_min": lo, "n_max": rng.randint(lo, 12),
                "precision": rng.choice(["mixed", "mixed", "fp64"])}
    if kind == "autograd":
        lo = rng.randint(1, 4)
        return {"kind": kind, "count": rng.randint(1, 8), "n_min": lo, "n_max": rng.randint(lo, 5)}
    if kind == "uhf":
        lo = rng.randint(1, 4)
        return {"kind": kind, "count": rng.randint(1, 12), "n_min": lo, "n_max": rng.randint(lo, 6),
                "precision": rng.choice(["mixed", "fp64"])}
    if kind == "fock":
        return {"kind": kind, "waters": rng.randint(1, 9)}
    waters = rng.randint(1, 16)
    # a group of equal molecules up to the listed cases' size
    most = {"integrals": 6000, "gradient": 2800, "whiten": 8000, "purify": 31000,
            "jk": 32768, "jk_increment": 13310}[kind] // waters ** 3
    return {"kind": kind, "waters": waters, "count": log_int(1, max(1, min(64, most)))}


# -- molecules and inputs ----------------------------------------------------


def _clusters(case, seed):
    """Sizes spread evenly over n_min..n_max (the same for every seed); geometries from the seed."""
    lo, hi, count = case["n_min"], case["n_max"], case["count"]
    sizes = [lo + i % (hi - lo + 1) for i in range(count)]
    make = geometry.alkane if case["kind"] == "autograd" else geometry.water_cluster
    return [make(n, np.random.default_rng([seed, i])) for i, n in enumerate(sizes)]


def _group(case, seed):
    """A native plan over equal clusters, and its coordinates on the device."""
    mols = [make_molecule(geometry.water_cluster(case["waters"], np.random.default_rng([seed, i])),
                          BASIS, AUX) for i in range(case["count"])]
    plan = NativePlan(mols, True)
    return plan, torch.as_tensor(plan.coordinates(), device="cuda").contiguous()


def _whitened(ints):
    """B = A L^-T (M = L L^T), packed rows, in plain FP64."""
    low = torch.linalg.cholesky(ints.metric)
    return torch.linalg.solve_triangular(low, ints.a_packed.transpose(1, 2), upper=False) \
        .transpose(1, 2).contiguous()


def _orthogonalizer(s):
    lam, vec = torch.linalg.eigh(s)
    return (vec * lam.rsqrt()[:, None, :]) @ vec.transpose(1, 2)


def _occupied(f, xo, nocc):
    """AO factor of the lowest orbitals, D = 2 C C^T, and the virtual ones."""
    c = xo @ torch.linalg.eigh(xo.transpose(1, 2) @ f @ xo)[1]
    return c[:, :, :nocc].contiguous(), c[:, :, nocc:].contiguous()


def _full(packed, n):
    """(N, N, X) rows of one molecule's packed pairs."""
    i = torch.arange(n, device=packed.device)
    hi, lo = torch.maximum(i[:, None], i), torch.minimum(i[:, None], i)
    return packed[hi * (hi + 1) // 2 + lo]


def _jk_plain(packed, c):
    """J and K of D = 2 C C^T for one molecule in FP64."""
    n, o = c.shape
    b = _full(packed, n)
    u = torch.einsum("mnq,ni->miq", b, c)
    rho = 2.0 * torch.einsum("mi,miq->q", c, u)
    u = u.reshape(n, -1)
    return (b.reshape(n * n, -1) @ rho).view(n, n), 2.0 * (u @ u.T)


def _density_inputs(case, seed):
    """Whitened tensor, core-guess orbitals and the matrices they came from."""
    plan, xyz = _group(case, seed)
    ints = scf.compute_integrals(plan, xyz)
    nocc = plan.layout[0].nocc
    b = _whitened(ints)
    xo = _orthogonalizer(ints.s)
    c, virt = _occupied(ints.h, xo, nocc)
    return plan, ints, b, xo, c, virt


def _nearby(c, virt, seed):
    """Orbitals of a density about 1e-5 away, as between late SCF iterations."""
    g = torch.Generator(device=c.device).manual_seed(seed)
    mix = torch.randn(c.shape[0], virt.shape[2], c.shape[2], generator=g, dtype=torch.float64,
                      device=c.device)
    return c + 1e-6 * (virt @ mix)


def _fock_input(case, seed):
    """F = H + J - K/2 of the core-guess density in the orthogonal basis, and n_occ."""
    plan, ints, b, xo, c, _ = _density_inputs(case, seed)
    f = ints.h.clone()
    for m in range(len(f)):
        j, k = _jk_plain(b[m], c[m])
        f[m] += 0.5 * (j - 0.5 * k)  # damped: the guess density overshoots
    fo = xo.transpose(1, 2) @ f @ xo
    return 0.5 * (fo + fo.transpose(1, 2)), c.shape[2]


def prepare(case, seed):
    kind = case["kind"]
    opts = dict(basis=BASIS, auxiliary_basis=AUX, device="cuda", density_fitting="cuda")
    if kind == "singlepoint":
        return {"case": case, "calc": Calculator(method="rhf", **opts),
                "atoms": geometry.water_cluster(case["waters"], np.random.default_rng([seed, 0]))}
    if kind in ("execute", "uhf"):
        systems = _clusters(case, seed)
        calc = Calculator(method="rhf" if kind == "execute" else "uhf", precision=case["precision"],
                          **opts)
        cation = {} if kind == "execute" else {"charges": [1] * len(systems),
                                               "multiplicities": [2] * len(systems)}
        return {"case": case, "batch": calc.prepare_batch(systems, warm_start=False, **cation),
                "coords": [np.array([p for _, p in s]) for s in systems]}
    if kind == "autograd":
        systems = _clusters(case, seed)
        calc = Calculator(method="rhf", **{**opts, "auxiliary_basis": AUX_CARBON})
        return {"case": case, "batch": calc.prepare_batch(systems, warm_start=False),
                "numbers": [[atomic_number(s) for s, _ in sys_] for sys_ in systems],
                "coords": [torch.tensor([p for _, p in sys_], dtype=torch.float64, device="cuda",
                                        requires_grad=True) for sys_ in systems]}
    if kind == "fock":
        one = {**case, "count": 1}
        plan, ints, _, _, c, _ = _density_inputs(one, seed)
        atoms = geometry.water_cluster(case["waters"], np.random.default_rng([seed, 0]))
        return {"case": case, "plan": FockPlan(atoms, BASIS, auxiliary_basis=AUX),
                "density": (2.0 * c[0] @ c[0].T).cpu().numpy()}
    if kind == "integrals":
        plan, xyz = _group(case, seed)
        return {"case": case, "plan": plan, "xyz": xyz}
    if kind == "gradient":
        plan, xyz = _group(case, seed)
        g = torch.Generator(device="cuda").manual_seed(seed)
        n, x = plan.layout[0].nao, plan.layout[0].naux
        weights = {k: torch.randn(size, generator=g, dtype=torch.float64, device="cuda")
                   for k, size in (("abar", plan.a_total), ("mbar", plan.met_total),
                                   ("dens", plan.mat_total), ("wdens", plan.mat_total))}
        for k, d in (("mbar", x), ("dens", n), ("wdens", n)):  # symmetric, as the energy's weights are
            m = weights[k].view(-1, d, d)
            weights[k] = (0.5 * (m + m.transpose(1, 2))).contiguous()
        return {"case": case, "plan": plan, "xyz": xyz, **weights}
    if kind == "whiten":
        plan, xyz = _group(case, seed)
        ints = scf.compute_integrals(plan, xyz)
        return {"case": case, "raw": ints.a_packed, "metric": ints.metric,
                "factor": scf.factor_metric(ints.metric), "work": torch.empty_like(ints.a_packed)}
    if kind == "purify":
        fo, nocc = _fock_input(case, seed)
        return {"case": case, "fo": fo, "nocc": nocc, "graphs": {}}
    plan, ints, b, xo, c, virt = _density_inputs(case, seed)
    n, x = c.shape[1], b.shape[2]
    builder = jkmod.make_builder("mixed", b, n, x, c.shape[2])
    if kind == "jk_increment":
        builder.anchor(2.0 * c @ c.transpose(1, 2), c)
        c = _nearby(c, virt, seed)
    return {"case": case, "jk": builder, "c": c, "d": 2.0 * c @ c.transpose(1, 2)}


# -- one pass ----------------------------------------------------------------


def run(state):
    kind = state["case"]["kind"]
    if kind == "singlepoint":
        r = state["calc"].singlepoint(state["atoms"])
        return {"energy": r.energy, "forces": r.forces}
    if kind in ("execute", "uhf"):
        items = state["batch"].execute(state["coords"], strict=True).items
        return {"energies": np.array([i.energy for i in items]),
                "forces": np.concatenate([i.forces for i in items])}
    if kind == "autograd":
        e = batched_energy(state["coords"], state["numbers"], prepared_batch=state["batch"])
        grads = torch.autograd.grad(e.sum(), state["coords"])
        return {"energies": e.detach(), "gradients": torch.cat(grads)}
    if kind == "fock":
        ev = state["plan"].evaluate(state["density"], derivative=True)
        return {"fock": ev.fock, "coulomb": ev.coulomb, "exchange": ev.exchange,
                "gradient": ev.gradient, "energy": ev.energy}
    if kind == "integrals":
        ints = scf.compute_integrals(state["plan"], state["xyz"])
        return {"s": ints.s, "h": ints.h, "metric": ints.metric, "a": ints.a_packed}
    if kind == "gradient":
        plan, xyz = state["plan"], state["xyz"].data_ptr()
        grad = torch.zeros(plan.natom, 3, dtype=torch.float64, device="cuda")
        st = torch.cuda.current_stream().cuda_stream
        _lib.call("vqc_grad1e", plan.handle, xyz, state["dens"].data_ptr(),
                  state["wdens"].data_ptr(), grad.data_ptr(), st)
        _lib.call("vqc_grad3c", plan.handle, xyz, state["abar"].data_ptr(), grad.data_ptr(), st)
        _lib.call("vqc_grad2c", plan.handle, xyz, state["mbar"].data_ptr(), grad.data_ptr(), st)
        return {"gradient": grad}
    if kind == "whiten":
        # the whitening is in place: the copy stands for the freshly made integrals
        state["work"].copy_(state["raw"])
        scf.whiten_tensor_cores(state["work"], state["factor"], state["metric"])
        return {"b": state["work"]}
    if kind == "purify":
        return {"projector": scf.purify_sp2(state["fo"], state["nocc"], graphs=state["graphs"])}
    if kind == "jk_increment":
        j, k, rho = state["jk"].build_incremental(state["d"], state["c"])
        return {"j": j, "k": k, "rho": rho}
    j, k = state["jk"].build(state["d"], state["c"])
    return {"j": j, "k": k}


# -- what a pass cannot do without, and how exact it is ----------------------


def _shape(waters):
    return 24 * waters, 116 * waters, 5 * waters  # N, X, n_occ


def _scf_work(n, x, o, precision_bytes):
    """Energy and forces of one molecule: the tensor written once, about 15 builds over it."""
    p = n * (n + 1) // 2
    builds = 15
    flops = p * x * x + builds * (2.0 * n * n * x * o + x * o * n * (n + 1) + 20.0 * n ** 3)
    return {"bytes": builds * p * x * precision_bytes, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind in ("singlepoint", "execute", "uhf", "autograd"):
        total = {"bytes": 0.0, "flops": 0.0}
        if kind == "singlepoint":
            sizes = [case["waters"]]
        else:
            sizes = [case["n_min"] + i % (case["n_max"] - case["n_min"] + 1)
                     for i in range(case["count"])]
        size = 4 if case.get("precision") == "mixed" else 8
        for k in sizes:
            n, x, o = _shape(k) if kind != "autograd" else (24 * k + 10, 43 * k + 12, 4 * k + 1)
            w = _scf_work(n, x, o, size)
            for key in total:
                total[key] += w[key] * (2 if kind == "uhf" else 1)
        return total
    n, x, o = _shape(case["waters"])
    p, nb = n * (n + 1) // 2, case.get("count", 1)
    if kind == "fock":
        return {"bytes": 8.0 * p * x * 2 + 8.0 * 4 * n * n,
                "flops": 4.0 * n * n * x + 4.0 * n ** 3 * x + 4.0 * n ** 3 * x + 1.0 * p * x * x}
    if kind == "integrals":  # about 100 operations an integral
        return {"bytes": nb * 8.0 * (p * x + x * x + 2 * n * n), "flops": nb * 100.0 * (p * x + x * x)}
    if kind == "gradient":  # six derivatives an integral
        return {"bytes": nb * 8.0 * (p * x + x * x + 2 * n * n), "flops": nb * 400.0 * (p * x + x * x)}
    if kind == "whiten":  # W is triangular
        return {"bytes": nb * (16.0 * p * x + 8.0 * x * x), "flops": nb * 1.0 * p * x * x}
    if kind == "purify":  # about 25 symmetric squarings
        return {"bytes": nb * 16.0 * n * n, "flops": nb * 25.0 * n ** 3}
    if kind == "jk":
        return {"bytes": nb * (4.0 * p * x + 8.0 * 3 * n * n),
                "flops": nb * (4.0 * p * x + 2.0 * n * n * x * o + x * o * n * (n + 1.0))}
    return {"bytes": nb * (4.0 * p * x + 8.0 * n * o * x + 8.0 * 3 * n * n),
            "flops": nb * (4.0 * p * x + 2.0 * n * n * x * o + 2 * x * o * n * (n + 1.0))}


def tolerance(case):
    kind = case["kind"]
    if kind in ("singlepoint", "execute", "uhf", "autograd"):
        # converged to 1e-10 Eh in the energy and 1e-8 in the density: forces
        # and gradients carry about the density's error
        return {"rel": 1e-6, "max": 1e-5}
    if kind in ("fock", "integrals"):
        return {"rel": 1e-11, "max": 1e-8}
    if kind == "gradient":
        return {"rel": 1e-10, "max": 1e-8}
    if kind == "whiten":  # 1.5e-11 off plain FP64
        return {"rel": 6e-11, "max": 1e-8}
    if kind == "purify":  # stops at tr X - tr X^2 < 1e-11
        return {"rel": 1e-11, "max": 1e-9}
    if kind == "jk_increment":  # K 2.5e-12 off plain FP64: the increment's split products
        return {"rel": 1e-11, "max": 1e-9}
    # K 1.7e-6 off plain FP64 (FP32 accumulation on the tensor cores), J 1.7e-8
    return {"rel": 7e-6, "max": 1e-4}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("jk", "jk_increment"):
        _, _, b, _, c, virt = _density_inputs(case, seed)
        if kind == "jk_increment":
            c = _nearby(c, virt, seed)
        js, ks = zip(*(_jk_plain(b[m], c[m]) for m in range(len(c))))
        out = {"j": torch.stack(js), "k": torch.stack(ks)}
        if kind == "jk_increment":
            out["rho"] = torch.stack([torch.einsum("mn,mnq->q", 2.0 * c[m] @ c[m].T,
                                                   _full(b[m], c.shape[1])) for m in range(len(c))])
        return out
    if kind == "whiten":
        plan, xyz = _group(case, seed)
        return {"b": _whitened(scf.compute_integrals(plan, xyz))}
    if kind == "purify":
        fo, nocc = _fock_input(case, seed)
        v = torch.linalg.eigh(fo)[1][:, :, :nocc]
        return {"projector": v @ v.transpose(1, 2)}
    # energies, forces and integrals have no plain form without integral code
    return None
