"""fesom_gpu_vdiff_impl_noalloc where its status page cannot be page-locked: the solve and its check of
the level bounds work as they do with it."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# A process of its own: the page is locked at the library's first call.  The test locks the page before
# that call, so the library's own attempt is refused (already registered).
CHILD = r"""
import ctypes as C, os, subprocess, sys
import numpy as np, torch
from fesom2_gb300 import gpu as G
from tests.test_zz_no_alloc import _case, _entry

torch.zeros(1, device="cuda")
L = G.load()
path = os.path.realpath(G.LIB_PATH)
off = [int(l.split()[0], 16) for l in subprocess.run(["nm", "-C", path], capture_output=True, text=True).stdout.splitlines()
       if l.endswith("g_host_status")]
assert len(off) == 1, off
base = min(int(l.split("-")[0], 16) for l in open("/proc/self/maps") if l.rstrip().endswith(path))
rt = torch.cuda.cudart()
assert int(rt.cudaHostRegister(base + off[0], 4096, 0)) == 0, "the test could not lock the page itself"

mesh, f, T0 = _case()
ctx = G.Context(mesh, G.PREC_FP64)
want = T0.copy()
ctx.vdiff_impl(f, G.tra_cfg(), want)
dev = lambda a, t: torch.as_tensor(np.ascontiguousarray(a, dtype=t), device="cuda")
nlev, ulev = dev(mesh.nlevels_nod2D, np.int32), dev(mesh.ulevels_nod2D, np.int32)
rest = [dev(a, np.float64) for a in (mesh.zbar_n_bot, mesh.hnode_new, mesh.area, mesh.areasvol, f.Kv, f.bc_surface)]
p = lambda t: C.c_void_p(t.data_ptr())
err = C.create_string_buffer(512)
def solve(lev):
    v = dev(T0, np.float64)
    rc = _entry()(mesh.nod2D, mesh.nl, p(lev), p(ulev), *[p(t) for t in rest], 600.0, p(v), None, err, 512)
    return rc, v.cpu().numpy()
rc, got = solve(nlev)
assert rc == 0, err.value
assert np.array_equal(got, want)
bad = nlev.clone()
bad[5] = mesh.nl + 1  # outside the mesh's levels: the kernel skips the column and reports it
assert solve(bad)[0] == 3, err.value
assert solve(nlev)[0] == 0
print("ok")
"""


@pytest.mark.gpu
def test_solve_without_a_page_locked_status_word():
    pytest.importorskip("torch")
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
