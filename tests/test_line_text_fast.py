"""The short ways of the line-list conversions (csrc/linefmt.h: a 64-bit power of ten for %E, a
128-bit product for %f) where they can go wrong: next to rounding boundaries, at the ends of
their ranges and between them and the big integers.  Every byte is compared with the C
library's printf, so there is no tolerance."""
import math

import numpy as np
import pytest

from test_line_text_cpu import c_printf


def _boundary_values(prec, seed):
    """Doubles on both sides of (D + 1/2) 10^k, D of prec + 1 digits, and of powers of ten."""
    rng = np.random.default_rng(seed)
    vals = []
    for X in list(range(-323, 309, 9)) + [-1, 0, 1]:
        lo = 10 ** prec
        for D in (lo, lo + 1, 10 * lo - 2, 10 * lo - 1, int(rng.integers(lo, 10 * lo))):
            x = float(f"{D}.5e{X - prec}")
            if x == 0.0 or math.isinf(x):
                continue
            vals += [x, math.nextafter(x, 0.0), math.nextafter(x, math.inf), -x]
        x = float(f"1e{X}")
        vals += [x, math.nextafter(x, 0.0), math.nextafter(x, math.inf)]
    return [v for v in vals if not math.isinf(v)]


def _fixed_values(seed):
    """m 2^-s over the shifts of the 128-bit product, and around 2^33, where it ends."""
    rng = np.random.default_rng(seed)
    vals = []
    for s in (0, 1, 19, 20, 21, 52, 53, 62, 63, 64, 65, 66, 80, 100, 126, 127, 128, 129, 300, 1074):
        for m in (2 ** 52, 2 ** 53 - 1, int(rng.integers(2 ** 52, 2 ** 53)), int(rng.integers(1, 2 ** 20))):
            vals.append(math.ldexp(float(m), -s))
    for c in (2.0 ** 33, 1e9, 1e9 - 0.5, 999999999.9999995, 2.0 ** 32):
        vals += [c, math.nextafter(c, 0.0), math.nextafter(c, math.inf), c - 0.5, c + 0.5]
    return vals + [-v for v in vals]


@pytest.mark.parametrize("prec", [0, 3, 9, 17])
def test_exponent_form_next_to_boundaries(built_lib, prec):
    import gainls
    vals = _boundary_values(prec, 5 + prec)
    bad = [x for x in vals if gainls.format_value(x, "E", 16, prec) != c_printf(f"%16.{prec}E", x)]
    assert not bad, bad[:10]


@pytest.mark.parametrize("prec", [0, 6, 9])
def test_fixed_form_over_the_shifts(built_lib, prec):
    import gainls
    vals = _fixed_values(3 + prec)
    bad = [x for x in vals if gainls.format_value(x, "f", 12, prec) != c_printf(f"%12.{prec}f", x)]
    assert not bad, bad[:10]


@pytest.mark.gpu
@pytest.mark.parametrize("conv,prec", [("E", 9), ("E", 17), ("f", 6)])
def test_device_next_to_boundaries(built_lib, conv, prec):
    import gainls
    vals = _boundary_values(prec, 9) + _fixed_values(9)
    got = gainls.format_values_device(vals, conv, 16, prec)
    bad = [x for x, a in zip(vals, got) if a != c_printf(f"%16.{prec}{conv}", x)]
    assert not bad, bad[:10]


@pytest.mark.gpu
@pytest.mark.parametrize("gns,n,host", [(-1.0, 40, False), (-1e-78, 40, True), (1e-78, 40, True), (-3.0, 13, True)])
def test_text_with_a_signed_intensity(built_lib, gns, n, host):
    """A negative spin weight gives the intensity a sign, and its field 17 characters where the
    exponent has three digits; with the positive one the field is always 16 wide.  Few columns
    and more than a block's lines, so rows begin inside a block."""
    import gainls
    import oracle
    import synth
    p = synth.make_problem(n, [2, 3], "c4", blocks=[(2, 0), (3, 1)])
    eng = gainls.Engine(11, p.nsym, 1)
    gainls.upload_problem(eng, p)
    bI, bF = p.blocks[(0, 0)], p.blocks[(1, 1)]
    lo, up = list(range(bI.vecs.shape[0])), list(range(0, bF.vecs.shape[0], 3))
    eng.run_pair(0, 0, 1, 1, lo, up, gainls.PATH_PLAIN_FP64)
    eI, eF = bI.energies[lo] + 0.0, bF.energies[up] + 0.0
    ref, nref = oracle.line_list(eng.fetch_amp(), eI, eF, lo, up, 2, 3, 0, 1, gnsF=gns)
    assert nref > 0
    if host:
        out = np.zeros(len(ref) + 64, np.uint8)
        text, k = eng.lines_text_host(eI, eF, 2, 3, 0, 1, out, gnsF=gns)
    else:
        text, k = eng.lines_text(eI, eF, 2, 3, 0, 1, gnsF=gns)
    assert k == nref and bytes(text) == ref
