"""GILA_KX_CHUNKS where it takes effect: read at the process's first matvec,
also when the operator was made before, and at y lengths of the tuned set whose y
passes are the mixed-radix ones (96, 192, 384).  Bit-identical to the unpipelined
run, in matvecs and in captured solver cycles; a child process each."""
from __future__ import annotations

import json
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as ct, json, os, sys
import numpy as np
import torch
sys.path.insert(0, {root!r}); sys.path.insert(0, {tests!r})
from conftest import load_pkg
from oracle.synth import seeded_current, synth_operator
gila = load_pkg()
SCL = ("1/32",) * 3
out, n = {{}}, {{}}
late = sys.argv[1] == "late"
mems = []
for k, (cel, dtype) in enumerate([((32, 48, 48), np.complex128), ((64, 96, 32), np.complex128),
                                  ((64, 48, 48), np.complex64), ((64, 192, 32), np.complex64)]):
    mix, fur, *_ = synth_operator(cel, SCL, (0, 0, 0), None, None)
    mems.append((cel, dtype, gila.GlaOprMem(gila.GlaKerOpt(True), gila.GlaVol(cel, SCL),
                                            egoFur=[f.astype(dtype) for f in fur], setTyp=dtype)))
G = gila.GlaOpr(gila.GlaOprMem(gila.GlaKerOpt(1.0 + 0j, 8, False, True, (), ()), gila.GlaVol((32, 48, 32), SCL)))
if late:
    os.environ["GILA_KX_CHUNKS"] = "4"
for k, (cel, dtype, mem) in enumerate(mems):
    xs = np.asfortranarray(np.stack([seeded_current(cel, s) for s in (1, 2)], axis=-1).astype(dtype))
    y = np.zeros_like(xs, order="F")
    mem.apply_into(xs, y, nrhs=2)
    out["y%d" % k], n["y%d" % k] = y, mem.launches_per_apply(2)
# the allocation-free entry point as an operator's first call
cel = (32, 48, 48)
mix, fur, *_ = synth_operator(cel, SCL, (0, 0, 0), None, None)
mem = gila.GlaOprMem(gila.GlaKerOpt(True), gila.GlaVol(cel, SCL), egoFur=fur, setTyp=np.complex128)
xt = torch.from_numpy(seeded_current(cel, 7).ravel(order="F").copy()).cuda()
yt = torch.zeros_like(xt)
torch.cuda.synchronize()
L = gila._lib
assert L.lib().gila_opr_apply_noalloc(mem._h, L.GILA_C128, ct.c_void_p(xt.data_ptr()), xt.numel(),
                                      ct.c_void_p(yt.data_ptr()), yt.numel(), None) == L.GILA_OK
out["noalloc"] = yt.cpu().numpy()
chi = np.zeros((32, 48, 32), dtype=np.complex128, order="F")
chi[8:24, 8:24, 8:24] = 2.0 + 0.1j
x, info = gila.solve(gila.LippmannSchwinger(G, chi), np.asfortranarray(seeded_current((32, 48, 32), 5)), mixed=True)
assert info.converged == 1
out["x"] = x
np.savez({path!r}, **out)
print(json.dumps(n))
"""


def _child(tmp_path, name, arg, env):
    path = str(tmp_path / f"{name}.npz")
    src = CHILD.format(root=ROOT, tests=os.path.join(ROOT, "tests"), path=path)
    base = {k: v for k, v in os.environ.items() if k != "GILA_KX_CHUNKS"}
    r = subprocess.run([sys.executable, "-c", src, arg], capture_output=True, text=True,
                       env=dict(base, GILA_AUTOTUNE="0", **env), timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1]), np.load(path)


def test_pipeline_setting_before_and_after_the_operator(tmp_path):
    n0, ref = _child(tmp_path, "off", "off", {})
    for name, arg, env in (("early", "off", {"GILA_KX_CHUNKS": "4"}), ("late", "late", {})):
        n, got = _child(tmp_path, name, arg, env)
        for k in n0:
            assert n[k] > n0[k], (name, k)
        for k in ref.files:
            assert np.array_equal(got[k], ref[k]), (name, k)
