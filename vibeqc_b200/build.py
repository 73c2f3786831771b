"""Build the sm_100a shared library ``libvqc_b200.so`` in-tree.

    python -m vibeqc_b200.build

Steps: generate ``csrc/sph_table.inc`` (Cartesian -> real-spherical transforms
from :mod:`vibeqc_b200.basis`), generate ``csrc/rys_table.inc`` when it is
missing (``csrc/gen_rys_table.py``), then compile every ``csrc/*.cu`` with nvcc
for ``sm_100a`` and link one shared library next to this file.
"""

from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
LIB = HERE / "libvqc_b200.so"
BUILD = HERE.parent / "_build"
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
KMAXL = 4


def gen_sph_table() -> Path:
    from vibeqc_b200 import basis as bas

    nc = (KMAXL + 1) * (KMAXL + 2) // 2
    ns = max(2 * KMAXL + 1, nc)  # Cartesian mode has ncart(l) output rows
    rows = []
    for mode in (0, 1):
        lblocks = []
        for l in range(KMAXL + 1):
            t = bas.transform_matrix(l, spherical=(mode == 0))
            block = []
            for r in range(ns):
                vals = [float(t[r, c]) if r < t.shape[0] and c < t.shape[1] else 0.0 for c in range(nc)]
                block.append("{" + ",".join(float.hex(v) for v in vals) + "}")
            lblocks.append("{" + ",\n".join(block) + "}")
        rows.append("{" + ",\n".join(lblocks) + "}")
    text = (
        "// Generated by vibeqc_b200/build.py from vibeqc_b200.basis: Cartesian (CCA order)\n"
        "// -> output functions; mode 0 real spherical (PySCF order), mode 1 normalised\n"
        "// Cartesian.  Included inside namespace vqc.\n"
        f"#define SPH_NS {ns}\n#define SPH_NC {nc}\n"
        f"static __constant__ double c_trans[2][{KMAXL + 1}][SPH_NS][SPH_NC] = {{\n"
        + ",\n".join(rows)
        + "};\n"
    )
    out = CSRC / "sph_table.inc"
    if not out.exists() or out.read_text() != text:
        out.write_text(text)
    return out


def _generator_grid() -> dict[str, str]:
    """LAYOUT, DEG and H as written in gen_rys_table.py."""
    grid = {}
    for line in (CSRC / "gen_rys_table.py").read_text().splitlines():
        name, _, value = line.partition(" = ")
        if name in ("LAYOUT", "DEG", "H"):
            grid[name] = value.split("#")[0].strip()
    return grid


def ensure_rys_table() -> Path:
    """Generate rys_table.inc when missing or written for another grid or layout."""
    out = CSRC / "rys_table.inc"
    stale = True
    if out.exists():
        head = out.read_text()[:2000]
        stale = any(f"#define RYS_{name} {value}\n" not in head
                    for name, value in _generator_grid().items())
    if stale:
        subprocess.run([sys.executable, str(CSRC / "gen_rys_table.py")], check=True)
    return out


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def build(verbose: bool = False, force: bool = False) -> Path:
    gen_sph_table()
    ensure_rys_table()
    BUILD.mkdir(exist_ok=True)
    deps = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.inc")) + list(
        (HERE.parent / "include").glob("*.h")
    )
    newest_dep = max(p.stat().st_mtime for p in deps)
    objs, jobs = [], []
    for src in sources():
        obj = BUILD / (src.stem + ".o")
        objs.append(obj)
        if not force and obj.exists() and obj.stat().st_mtime > max(src.stat().st_mtime, newest_dep):
            continue
        cmd = [
            NVCC, *ARCH, "-O3", "-lineinfo", "-std=c++17", "--expt-relaxed-constexpr",
            "-Xcompiler", "-fPIC", "-I", str(CSRC), "-I", str(HERE.parent / "include"),
            "-c", str(src), "-o", str(obj),
        ]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        jobs.append((src.name, cmd))
    procs = []
    for name, cmd in jobs:  # translation units compile concurrently
        print("nvcc", name, flush=True)
        procs.append((name, subprocess.Popen(cmd)))
    failed = [name for name, p in procs if p.wait() != 0]
    if failed:
        raise RuntimeError(f"nvcc failed for {failed}")
    link = [NVCC, *ARCH, "-shared", "-o", str(LIB), *map(str, objs)]
    subprocess.run(link, check=True)
    return LIB


if __name__ == "__main__":
    build(verbose="-v" in sys.argv, force="-f" in sys.argv)
    print(LIB)
