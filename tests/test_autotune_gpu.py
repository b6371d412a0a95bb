"""What the autotuner times for an operator (GILA_TUNE_DEBUG lists it)."""
from __future__ import annotations

import re

import numpy as np
import pytest

from conftest import load_pkg, rel_l2, TOL_F32, TOL_F64
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
