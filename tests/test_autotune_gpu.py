"""What the autotuner times for an operator (GILA_TUNE_DEBUG lists it)."""
from __future__ import annotations

import os
import re
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, TOL_F32, TOL_F64, load_pkg, rel_l2
from oracle.matvec import OprMem, ego_opr
from oracle.synth import seeded_current, synth_operator

pytestmark = pytest.mark.gpu

SCL = ("1/32", "1/32", "1/32")


def _operator(gila, cel, dtype):
    mix, fur, *_ = synth_operator(cel, SCL, (0, 0, 0), None, None, set_dtype=np.complex128)
    fur = [f.astype(dtype) for f in fur]
    mem = gila.GlaOprMem(gila.GlaKerOpt(True), gila.GlaVol(cel, SCL), None, egoFur=fur, setTyp=dtype)
    return mix, mem, OprMem(mix, [f.astype(np.complex128) for f in fur])


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64], ids=["c128", "c64"])
@pytest.mark.parametrize("cel", [(32, 48, 8), (64, 10, 8), (32, 32, 8)], ids=lambda c: "x".join(map(str, c)))
def test_xy_form_is_timed_wherever_x_has_both(cel, dtype, monkeypatch, capfd):
    """x lengths 64 and 128 with y lengths that have tile variants (64) and
    that have none (96, 20): both forms of the x passes are candidates."""
    gila = load_pkg()
    mix, mem, ref = _operator(gila, cel, dtype)
    monkeypatch.setenv("GILA_TUNE_DEBUG", "1")
    capfd.readouterr()
    mem.autotune(1)
    seen = re.findall(r"global-fed x/y (\d)", capfd.readouterr().err)
    assert {"0", "1"} <= set(seen)
    x = np.asfortranarray(seeded_current(mix.src_cel, 3).astype(dtype))
    tol = TOL_F64 if dtype == np.complex128 else TOL_F32
    assert rel_l2(gila.egoOpr(mem, x), ego_opr(ref, x.astype(np.complex128))) <= tol


def test_c64_z64_has_one_tile_and_is_not_timed(monkeypatch, capfd):
    """The ComplexF32 z pass at 64 has one launch shape: nothing to time, and a
    tile width that it cannot take is not reported as taken.  In ComplexF64 every
    width is."""
    gila = load_pkg()
    monkeypatch.setenv("GILA_TUNE_DEBUG", "1")
    for dtype, widths in ((np.complex64, [16, 16, 16]), (np.complex128, [4, 8, 16])):
        _, mem, _ = _operator(gila, (8, 32, 32), dtype)
        capfd.readouterr()
        mem.autotune(1)
        assert ("z tile" in capfd.readouterr().err) == (dtype == np.complex128)
        got = []
        for w in (4, 8, 16):
            mem.tiles = (0, 0, 0, w)
            got.append(mem.tiles[3])
        assert got == widths


CHILD = r"""
import sys
import numpy as np
sys.path.insert(0, {root!r}); sys.path.insert(0, {tests!r})
from test_autotune_gpu import _operator
from conftest import load_pkg
from oracle.synth import seeded_current
gila = load_pkg()
mix, mem, ref = _operator(gila, (8, 32, 32), np.complex64)
np.save({path!r}, gila.egoOpr(mem, np.asfortranarray(seeded_current(mix.src_cel, 3).astype(np.complex64))))
"""


def test_c64_z64_honours_the_kernel_switches(tmp_path):
    """GILA_ZG=0 and GILA_ZFUSE=0 select other forms of the tuned z pass, which
    round differently, at every tuned length (each read once per process)."""
    out = {}
    for name, env in (("default", {}), ("zg", {"GILA_ZG": "0"}), ("zfuse", {"GILA_ZFUSE": "0"})):
        path = str(tmp_path / f"{name}.npy")
        src = CHILD.format(root=ROOT, tests=os.path.join(ROOT, "tests"), path=path)
        r = subprocess.run([sys.executable, "-c", src], capture_output=True, text=True,
                           env=dict(os.environ, **env), timeout=300)
        assert r.returncode == 0, r.stderr[-3000:]
        out[name] = np.load(path)
    for name in ("zg", "zfuse"):
        assert not np.array_equal(out[name], out["default"])
        assert rel_l2(out[name], out["default"]) <= TOL_F32
