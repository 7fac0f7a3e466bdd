"""The library in a second context of one process (what a second device is to it): nothing that
belongs to a context, such as a kernel's shared-memory limit, is remembered from the first."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# Each form in two contexts of the driver API, through the C entry points and the driver's own
# allocations alone (torch would make its primary context current). Prints the energies.
CHILD = r"""
import contextlib, ctypes, sys
import numpy as np
import torch
torch.cuda.device = lambda d: contextlib.nullcontext()
from fourierd3_b200 import _native, engine, geometry, structures

cu = ctypes.CDLL("libcuda.so.1")
vp, sz = ctypes.c_void_p, ctypes.c_size_t
cu.cuMemAlloc_v2.argtypes = [ctypes.POINTER(vp), sz]
cu.cuMemcpyHtoD_v2.argtypes = [vp, vp, sz]
cu.cuMemcpyDtoH_v2.argtypes = [vp, vp, sz]
cu.cuCtxCreate_v2.argtypes = [ctypes.POINTER(vp), ctypes.c_uint, ctypes.c_int]

def ok(rc):
    assert rc == 0, rc

def alloc(n):
    p = vp()
    ok(cu.cuMemAlloc_v2(ctypes.byref(p), n))
    return p

def upload(a):
    p = alloc(a.nbytes)
    ok(cu.cuMemcpyHtoD_v2(p, a.ctypes.data, a.nbytes))
    return p

ok(cu.cuInit(0))
lib = _native.lib()
boxes = {"few": (structures.random_box(seed=1, n_atoms=90, z_max=2), 0.3),    # 64^3: the x-passes apply
         "many": (structures.random_box(seed=2, n_atoms=90, z_max=30), 0.9)}
forms = [("few", "mixed", {}), ("few", "mixed", dict(fft_x=1)), ("few", "mixed", dict(gather_tile=1)),
         ("few", "fp64", {}), ("many", "mixed", {}), ("many", "mixed", dict(filter_kt=8)),
         ("many", "mixed", dict(filter_mma=1)), ("many", "fp64", {})]
for turn in range(2):
    ctx = vp()
    ok(cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, 0))
    for box, precision, knobs in forms:
        (pos, cell, numbers), spacing = boxes[box]
        h = np.ascontiguousarray(cell, dtype=np.float64).reshape(9)
        mesh = geometry.ns_mesh(np.asarray(cell) * geometry.ANGSTROM_TO_BOHR, spacing * geometry.ANGSTROM_TO_BOHR)
        eng = engine.Engine(engine.species_setup(np.asarray(numbers), 1.0), method="spme", order=4, mesh=mesh,
                            ewald_ns=(0, 0, 0), precision=precision, r_cut_bohr=6.0 * geometry.ANGSTROM_TO_BOHR,
                            params=engine.PBE_BJ, device=torch.device("cuda:0"))
        eng.set_tuning(**knobs)
        assert box == "many" or eng.tuning()["fft_x"] == knobs.get("fft_x", 2 if precision == "mixed" else 1)
        n = len(numbers)
        size = eng.workspace_bytes(n, h, 6.0)
        out, species = alloc(8 * (1 + 3 * n + 9)), upload(np.ascontiguousarray(eng.setup.species, dtype=np.int32))
        x = upload(np.ascontiguousarray(pos, dtype=np.float64))
        e = np.zeros(1)
        rc = lib.fd3_energy_forces_stress_hostcell(eng._plan, n, x, species, _native.dptr(h), 6.0, alloc(size), size,
                                                   out, out.value + 8, out.value + 8 + 24 * n, None)
        _native.check(rc, f"turn {turn} {box} {precision} {knobs}")
        ok(cu.cuMemcpyDtoH_v2(e.ctypes.data, out, 8))
        print(turn, box, precision, *knobs, e[0].hex())
        del eng
"""


def test_every_form_runs_in_a_second_context(cuda_device):
    run = subprocess.run([sys.executable, "-c", CHILD], cwd=REPO, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout + run.stderr
    lines = [line.split() for line in run.stdout.splitlines()]
    first = [line[1:] for line in lines if line[0] == "0"]
    assert len(first) == 8 and first == [line[1:] for line in lines if line[0] == "1"]
