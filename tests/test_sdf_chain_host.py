"""Compiled left folds on the host: the library's table builder (sdf_skip.hpp
sdf_chain_tables) next to a host restatement of the device's compiled
evaluation (tests/sdf_chain_check.cpp). At every march point the value equals
the full program's bit for bit (inner grid, outer grid and outside both), every
march returns the same hit and t with the escape exits, also for rays that
begin inside, and programs that are no left folds are not compiled."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from myrt_b200 import sdf as S

ROOT = Path(__file__).resolve().parent.parent


def _fold(nodes, op):
    acc = nodes[0]
    for i, nd in enumerate(nodes[1:]):
        acc = op(i, acc, nd)
    return acc


def _programs():
    """(name, node, compiled)."""
    rng = np.random.default_rng(8)

    def prim(i):
        kind = i % 4
        if kind == 0:
            return S.sphere(float(rng.uniform(0.03, 0.12)))
        if kind == 1:
            return S.box(tuple(rng.uniform(0.0, 0.1, 3)))
        if kind == 2:
            return S.torus(float(rng.uniform(0.05, 0.12)), float(rng.uniform(0.01, 0.04)))
        return S.vertical_capsule(float(rng.uniform(0.0, 0.2)), float(rng.uniform(0.02, 0.05)))

    def smooth(k):
        return lambda i, a, b: S.smooth_union(a, b, k)

    placed = [S.translate(prim(i), rng.uniform(-0.8, 0.8, 3)) for i in range(37)]
    out = [("chain256", S.random_sdf_field(256, k=0.1, seed=9, extent=0.8, chain=True), True),
           ("chain8", S.random_sdf_field(8, k=0.05, seed=2, extent=0.5, chain=True), True),
           ("mixed", _fold(placed, lambda i, a, b: S.union(a, b) if i % 3 == 0 else S.smooth_union(a, b, 0.07)), True)]
    big = [S.sphere(1.5)] + [S.translate(S.sphere(0.2), rng.uniform(-1.2, 1.2, 3)) for _ in range(20)]
    out.append(("big_sphere", _fold(big, smooth(0.2)), True))  # most rays begin inside; an untranslated primitive
    cluster = [S.translate(S.sphere(0.1 + float(rng.uniform(-1e-4, 1e-4))), rng.uniform(-1e-3, 1e-3, 3))
               for _ in range(33)]
    out.append(("cluster", _fold(cluster, smooth(0.2)), True))
    twice = [S.translate(S.translate(S.sphere(0.1), rng.uniform(-0.5, 0.5, 3)), (0.1, 0.0, 0.0)) for _ in range(12)]
    out.append(("two_translations", _fold(twice, smooth(0.1)), False))
    out.append(("tree", S.random_sdf_field(64, k=0.1, seed=5, extent=0.8, chain=False), False))
    return out


@pytest.mark.parametrize("cells", [8, 32])
def test_compiled_folds_are_exact(tmp_path, cells):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "sdf_chain_check"
    subprocess.run([gxx, "-O2", "-std=c++20", "-pthread", "-ffp-contract=off", "-I", "/usr/local/cuda/include",
                    "-o", str(exe), str(ROOT / "tests" / "sdf_chain_check.cpp")], check=True)
    progs = _programs()
    lib = S.SdfLibrary()
    for _, node, _ in progs:
        lib.add(node)
    np.asarray(lib.instrs, np.int32).tofile(tmp_path / "instrs.bin")
    np.asarray(lib.programs, np.int32).tofile(tmp_path / "programs.bin")
    np.asarray(lib.params, np.float32).tofile(tmp_path / "params.bin")
    res = subprocess.run([str(exe), str(tmp_path), str(cells), "900", "5"], check=True, capture_output=True, text=True)
    rows = [list(map(float, r.split())) for r in res.stdout.split("\n") if r.strip()]
    assert len(rows) == len(progs)
    began_inside = 0
    for (name, _, compiled), (groups, points, bad, outer, marches, hits, bad_marches, inside, _) in zip(progs, rows):
        assert (groups > 0) == compiled, name
        if not compiled:
            continue
        assert bad == 0 and bad_marches == 0, name
        assert points > 2000 and outer > 100 and marches > 800 and hits > 20, (name, points, outer, marches, hits)
        began_inside += inside
    assert began_inside > 50
