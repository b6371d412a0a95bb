"""GPU matvec parity at the mixed-radix lengths (every even 2^a 3^b 5^c 7^d up
to 512 without a tuned kernel), each length on each axis, against the FP64
oracle on the same kernel values; tolerances of the parity tests."""
from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

from conftest import TOL_F32, TOL_F64, load_pkg, rel_l2
from oracle.matvec import OprMem, ego_opr
from oracle.synth import seeded_current, synth_operator

pytestmark = pytest.mark.gpu

SCL = ("1/32", "1/32", "1/32")


def _smooth(n):
    for q in (2, 3, 5, 7):
        while n % q == 0:
            n //= q
    return n == 1


LENGTHS = [n for n in range(4, 513, 2) if _smooth(n) and n not in (64, 96, 128, 192, 256, 384, 512)]


def _operator(gila, tc, sc, to, dtype):
    mix, fur, *_ = synth_operator(tc, SCL, to, sc, None if sc is None else (0, 0, 0), set_dtype=np.complex128)
    sv = None if sc is None else gila.GlaVol(sc, SCL, (0, 0, 0))
    mem = gila.GlaOprMem(gila.GlaKerOpt(True), gila.GlaVol(tc, SCL, to), sv,
                         egoFur=[f.astype(dtype) for f in fur], setTyp=dtype)
    return mix, mem, OprMem(mix, [f.astype(dtype).astype(np.complex128) for f in fur])


@pytest.mark.parametrize("P", LENGTHS)
@pytest.mark.parametrize("dtype", [np.complex128, np.complex64], ids=["c128", "c64"])
def test_mx_lengths_each_axis(P, dtype):
    """Self where P is 4 n, else source and target of different extents (one
    of them more than half of the padded line); two vectors in one call."""
    import torch
    gila = load_pkg()
    for axis in range(3):
        if P % 4 == 0:
            tc, sc, to = [4, 4, 4], None, (0, 0, 0)
            tc[(axis + 1) % 3] = 6
            tc[axis] = P // 2
        else:
            a = max(2, P // 6 * 2)
            tc, sc, to = [4, 4, 4], [4, 4, 4], [0, 0, 0]
            tc[axis], sc[axis] = (a, P - a) if axis % 2 else (P - a, a)
            to[axis] = f"{P // 2 + 3}/32"
            to = tuple(to)
        mix, mem, ref = _operator(gila, tuple(tc), None if sc is None else tuple(sc), to, dtype)
        xs = [seeded_current(mix.src_cel, 31 + k).astype(dtype) for k in range(2)]
        X = np.asfortranarray(np.stack(xs, axis=-1))
        Xd = torch.from_numpy(np.ascontiguousarray(X.transpose(4, 3, 2, 1, 0))).cuda()
        Yd = mem.new_output(Xd, 2)
        mem.apply_into(Xd, Yd, nrhs=2)
        tol = TOL_F64 if dtype == np.complex128 else TOL_F32
        for k in range(2):
            got = Yd[k].cpu().numpy().transpose(3, 2, 1, 0)
            assert rel_l2(got, ego_opr(ref, xs[k].astype(np.complex128))) <= tol, (P, axis)


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64], ids=["c128", "c64"])
def test_mx_odd_row_counts_and_axpby(dtype):
    """Slab pieces of one plane and the fused axpby on mixed-radix lengths."""
    import torch
    gila = load_pkg()
    mix, mem, ref = _operator(gila, (30, 18, 10), None, (0, 0, 0), dtype)
    x = np.asfortranarray(seeded_current(mix.src_cel, 5).astype(dtype))
    o = np.asfortranarray(seeded_current(mix.trg_cel, 6).astype(dtype))
    want = (0.5 - 2j) * ego_opr(ref, x.astype(np.complex128)) + (0.25 + 1j) * o.astype(np.complex128)
    out = o.copy(order="F")
    gila.mul(out, gila.GlaOpr(mem), x, 0.5 - 2j, 0.25 + 1j)
    tol = TOL_F64 if dtype == np.complex128 else TOL_F32
    assert rel_l2(out, want) <= tol
    xd = torch.from_numpy(np.ascontiguousarray(x.transpose(3, 2, 1, 0))).cuda()
    yd = torch.empty_like(xd)
    mem.apply_into(xd, yd)
    for ranks in (3, 10):
        ys = gila.slab_apply_local(gila.SlabPieces(mem), xd, ranks)
        assert torch.equal(ys.reshape(yd.shape), yd)


def test_mx_unaligned_pairs():
    """ComplexF32 spectra on an 8-byte boundary (a slab piece's caller may
    hold its planes anywhere): the calls that were taken before, to rounding."""
    import torch
    gila = load_pkg()
    L = gila._lib
    mix, mem, _ = _operator(gila, (10, 12, 18), None, (0, 0, 0), np.complex64)
    Px, Py = 20, 24
    x = torch.from_numpy(np.ascontiguousarray(
        seeded_current(mix.src_cel, 9).astype(np.complex64).transpose(3, 2, 1, 0))).cuda()
    n = 3 * 18 * Px * Py
    outs = []
    for shift in (0, 1):
        b = torch.zeros(n + 2, dtype=torch.complex64, device="cuda")
        y = torch.empty_like(x)
        p = ct.c_void_p(b.data_ptr() + 8 * shift)
        torch.cuda.synchronize()
        for st in (L.lib().gila_opr_slab_fwd(mem._h, L.GILA_C64, ct.c_void_p(x.data_ptr()), 18, p, None),
                   L.lib().gila_opr_slab_z(mem._h, L.GILA_C64, p, 0, Py, None),
                   L.lib().gila_opr_slab_inv(mem._h, L.GILA_C64, p, 18, ct.c_void_p(y.data_ptr()), None)):
            assert st == L.GILA_OK
        outs.append(y.cpu().numpy())
    assert rel_l2(outs[1], outs[0]) <= TOL_F32
