"""ComplexF32 spectra on an 8-byte boundary: a slab piece's caller may hold its
planes on any element boundary, where the tuned lengths' line-pair kernels
(16-byte accesses) do not apply and the one-line kernels run instead."""
from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

from conftest import TOL_F32, load_pkg, rel_l2
from oracle.matvec import OprMem, ego_opr
from oracle.synth import seeded_current, synth_operator

pytestmark = pytest.mark.gpu

SCL = ("1/32", "1/32", "1/32")

# target cells, source cells and target origin (None: self); y and z lengths
CASES = [
    ((10, 32, 32), None, (0, 0, 0)),  # 64, 64
    ((10, 64, 48), None, (0, 0, 0)),  # 128, 96
    ((6, 128, 64), None, (0, 0, 0)),  # 256, 128
    ((6, 256, 96), None, (0, 0, 0)),  # 512, 192
    ((6, 48, 192), None, (0, 0, 0)),  # 96, 384
    ((6, 96, 128), None, (0, 0, 0)),  # 192, 256
    ((4, 8, 256), None, (0, 0, 0)),  # 16, 512
    ((6, 12, 16), (6, 20, 48), (0, 0, "50/32")),  # 32, 64: more than half of the line filled
    ((6, 20, 16), (6, 44, 80), (0, 0, "60/32")),  # 64, 96
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}<-{c[1]}")
@pytest.mark.parametrize("order", [0, 1])
def test_unaligned_planes_at_tuned_lengths(case, order):
    """Vectors and planes both eight bytes past a 16-byte boundary, against
    the aligned call (to rounding) and the oracle."""
    import torch
    gila = load_pkg()
    L = gila._lib
    tc, sc, to = case
    mix, fur, *_ = synth_operator(tc, SCL, to, sc, None if sc is None else (0, 0, 0), set_dtype=np.complex128)
    fur = [f.astype(np.complex64) for f in fur]
    sv = None if sc is None else gila.GlaVol(sc, SCL, (0, 0, 0))
    mem = gila.GlaOprMem(gila.GlaKerOpt(True), gila.GlaVol(tc, SCL, to), sv, egoFur=fur, setTyp=np.complex64)
    mem.schedule = (order, order)
    s = mix.src_cel
    Px, Py = s[0] + tc[0], s[1] + tc[1]
    xh = seeded_current(s, 9).astype(np.complex64)
    nx, ny, nb = 3 * int(np.prod(s)), 3 * int(np.prod(tc)), 3 * max(s[2], tc[2]) * Px * Py
    outs = []
    for shift in (0, 1):
        x = torch.zeros(nx + 2, dtype=torch.complex64, device="cuda")
        x[shift:shift + nx] = torch.from_numpy(np.ascontiguousarray(xh.transpose(3, 2, 1, 0)).ravel()).cuda()
        b = torch.zeros(nb + 2, dtype=torch.complex64, device="cuda")
        y = torch.zeros(ny + 2, dtype=torch.complex64, device="cuda")
        px, pb, py = (ct.c_void_p(t.data_ptr() + 8 * shift) for t in (x, b, y))
        torch.cuda.synchronize()
        for st in (L.lib().gila_opr_slab_fwd(mem._h, L.GILA_C64, px, s[2], pb, None),
                   L.lib().gila_opr_slab_z(mem._h, L.GILA_C64, pb, 0, Py, None),
                   L.lib().gila_opr_slab_inv(mem._h, L.GILA_C64, pb, tc[2], py, None)):
            assert st == L.GILA_OK
        assert not b[:shift].any() and not y[:shift].any() and not y[shift + ny:].any()
        outs.append(y[shift:shift + ny].cpu().numpy().reshape(3, tc[2], tc[1], tc[0]).transpose(3, 2, 1, 0))
    assert rel_l2(outs[1], outs[0]) <= TOL_F32
    ref = OprMem(mix, [f.astype(np.complex128) for f in fur])
    assert rel_l2(outs[1], ego_opr(ref, xh.astype(np.complex128))) <= TOL_F32
