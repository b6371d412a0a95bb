"""The radix orders of the x and y transforms: two at lengths 128 and 256 (8 8 2
and 8 8 4 and their reverses), one elsewhere."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import TOL_F32, TOL_F64, load_pkg, rel_l2
from oracle.matvec import OprMem, ego_opr
from oracle.synth import seeded_current, synth_operator

pytestmark = pytest.mark.gpu

SCL = ("1/32", "1/32", "1/32")


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64], ids=["c128", "c64"])
@pytest.mark.parametrize("cel,two", [((64, 128, 4), (True, True)), ((128, 64, 4), (True, True)),
                                     ((32, 256, 4), (False, False)), ((48, 96, 4), (False, False)),
                                     ((192, 64, 4), (False, True)), ((20, 50, 4), (False, False))],
                         ids=lambda v: "x".join(map(str, v)))
def test_orders(cel, two, dtype):
    gila = load_pkg()
    mix, fur, *_ = synth_operator(cel, SCL, (0, 0, 0), None, None, set_dtype=np.complex128)
    fur = [f.astype(dtype) for f in fur]
    mem = gila.GlaOprMem(gila.GlaKerOpt(True), gila.GlaVol(cel, SCL), None, egoFur=fur, setTyp=dtype)
    ref = OprMem(mix, [f.astype(np.complex128) for f in fur])
    x = np.asfortranarray(seeded_current(mix.src_cel, 23).astype(dtype))
    want = ego_opr(ref, x.astype(np.complex128))
    out = {}
    for sched in ((0, 0), (1, 0), (0, 1)):
        mem.schedule = sched
        assert mem.schedule == sched
        out[sched] = gila.egoOpr(mem, x)
        assert rel_l2(out[sched], want) <= (TOL_F64 if dtype == np.complex128 else TOL_F32)
    for k, sched in enumerate(((1, 0), (0, 1))):
        assert np.array_equal(out[sched], out[(0, 0)]) == (not two[k])
