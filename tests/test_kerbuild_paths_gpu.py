"""The GPU kernel build where its paths split: real and complex frequencies,
phases past the small-phase sums, cells with equal and unequal sides (repeated
weak integrals are evaluated once), fields of more items than one chunk."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_pkg
from oracle import kerbuild as kb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scl", [("1/32", "1/32", "1/32"), ("1/20", "1/25", "1/20"), ("1/2", "1/3", "1/2"),
                                 ("1/40", "1/2", "1/7")], ids=lambda s: "x".join(v.replace("/", "-") for v in s))
@pytest.mark.parametrize("frq", [1.0 + 0j, 0.8 + 0j, 1.0 + 0.125j], ids=["1", "0.8", "1+i8"])
def test_weak_integrals_by_frequency(scl, frq):
    """Same nodes and integrands on both sides: rounding of sums of up to
    24 * 12^3 terms times the kernel's 1 / d, 1e-11 of the largest value."""
    gila = load_pkg()
    got = np.concatenate(gila.weak_integrals(scl, frq, 12))
    ref = np.concatenate([np.asarray(v) for v in kb.weak(scl, frq, 12)])
    assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()


@pytest.mark.parametrize("frq", [1.0 + 0j, 0.9 + 0.05j], ids=["1", "0.9+i20"])
@pytest.mark.parametrize("scl", [("1/3", "1/2", "1/3"), ("1/30", "1/24", "1/27")], ids=["coarse", "fine"])
def test_external_build_by_frequency(scl, frq):
    """Separated volumes: pairs that converge at once and pairs refined in
    each of the region stores; the tolerance of the build's parity tests."""
    gila = load_pkg()
    num, den = (int(v) for v in scl[0].split("/"))
    to = (f"{4 * num}/{den}", 0, 0)
    mix, fur_ref, _, _, trg, src = kb.build_operator((2, 4, 2), scl, to, (4, 2, 2), (0, 0, 0), frq=frq, int_ord=8)
    opt = gila.GlaKerOpt(frq, 8, False, True, (), ())
    mem = gila.GlaOprMem(opt, gila.GlaVol(trg.cel, trg.scl, trg.org), gila.GlaVol(src.cel, src.scl, src.org))
    scale = max(np.abs(f).max() for f in fur_ref)
    assert max(np.abs(a - b).max() for a, b in zip(mem.egoFur, fur_ref)) <= 1e-9 * scale


@pytest.mark.parametrize("cel", [(36, 32, 32), (35, 30, 36)])
def test_chunked_field_matches_a_separate_pair(cel):
    """A self field of more than 2^15 offsets: the response at the far corner
    to currents in the near one against an external operator of the two
    corners, which lists and chunks its items differently."""
    gila = load_pkg()
    scl = ("1/32",) * 3
    opt = gila.GlaKerOpt(1.0 + 0j, 8, False, True, (), ())
    G = gila.GlaOprMem(opt, gila.GlaVol(cel, scl))
    x = np.zeros((*cel, 3), dtype=np.complex128, order="F")
    rng = np.random.default_rng(3)
    xs = rng.standard_normal((2, 2, 2, 3)) + 1j * rng.standard_normal((2, 2, 2, 3))
    x[:2, :2, :2] = xs
    y = gila.egoOpr(G, x)[-2:, -2:, -2:]
    E = gila.GlaOprMem(opt, gila.GlaVol((2, 2, 2), scl, tuple(f"{n - 2}/32" for n in cel)),
                       gila.GlaVol((2, 2, 2), scl))
    ye = gila.egoOpr(E, np.asfortranarray(xs))
    # the FFTs' rounding is of the whole field's scale, the corner's values
    # are about 1e-4 of it
    assert np.abs(y - ye).max() <= 1e-11 * np.abs(gila.egoOpr(G, x)).max()
