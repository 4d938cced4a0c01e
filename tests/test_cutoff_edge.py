"""Pairs at the Coulomb cutoff to the last bits, FP64: the reference keeps a pair
whose rounded dsqrt(r^2) is at most rrcut.  Two molecules are placed so that one
pair of oxygens lies at rrcut exactly (r^2 the rounded square of rrcut, or the
next double, whose root still rounds to rrcut), on a 2^-40 A grid, where every
difference is exact whatever the frame.  Bars: forces 1e-12 as
tests/test_pair_segments.py (the pair's own force is 1e-6 of the largest), the
record 1e-9 as tests/test_flux_sums.py, where the pair is a whole 1/r."""
import math
from fractions import Fraction

import numpy as np
import pytest

from tests.conftest import rel_rms
from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu

GRID = 2.0 ** 40


def _edge(nside, rr, dy):
    """nside^3 waters 6.4 A apart, the second molecule's oxygen at (rr, dy, 0) from the first's."""
    s = S.small_box("water", nside=nside, spacing=6.4, nfft=16, rcut=rr)
    s.params.update(rcut=rr + 0.5, rrcut=rr, rcut_book=rr + 2.5, alpha=2.0 / rr)   # alpha: the pair shows in the force
    x = np.rint(s.atmcor * GRID) / GRID
    first = s.molept_list[s.molept_index[:-1]]
    b = int(np.argmin(np.where(np.arange(len(first)) == 0, 1e9, np.linalg.norm(x[first] - x[first[0]] - [6.4, 0, 0], axis=1))))
    atoms = s.molept_list[s.molept_index[b]:s.molept_index[b + 1]]
    x[atoms] += x[first[0]] + [rr, dy, 0.0] - x[first[b]]
    s.atmcor[:] = x
    return s


def _kept(rr, dy):
    """dsqrt(r^2) <= rrcut with r^2 rounded once (fused) and after each operation; None where they decide differently."""
    x, y = Fraction(rr), Fraction(dy)
    r2 = {float(x * x + Fraction(float(y * y))), float(Fraction(float(x * x)) + Fraction(float(y * y))),
          float(Fraction(float(x * x)) + y * y)}
    got = {math.sqrt(v) <= rr for v in r2}
    return got.pop() if len(got) == 1 else None


# r^2 in [16, 32): its doubles are closer than those whose root is next to rrcut, so the next one can round to rrcut
CASES = [c for r in np.linspace(4.35, 5.6, 24) for dy in (0.0, 6.0e-8)
         for c in [(float(np.rint(r * GRID) / GRID), float(np.rint(dy * GRID) / GRID))] if _kept(*c) is not None]
assert sum(_kept(*c) for c in CASES) > 24 < len(CASES)


@pytest.mark.parametrize("nside", [4, 8])            # per-pair image; cluster frame
def test_pair_kernel_keeps_the_pair_at_the_cutoff(oracle_mod, nside):
    from thrid_b200.pgk import PgkEngine
    for rr, dy in CASES[:: 1 if nside == 4 else 4]:
        s = _edge(nside, rr, dy)
        o = oracle_mod.Oracle(s, threads=8)
        o.mklist()
        e = PgkEngine(s)
        e.mklist_cell()
        assert rel_rms(e.ewaldr()[0], o.ewaldrp()[0]) <= 1e-12, (rr, dy)
        e.close()


def test_record_and_arrays_keep_the_pair_at_the_cutoff(oracle_mod):
    from thrid_b200.pgk import PgkEngine
    for rr, dy in CASES:
        s = _edge(4, rr, dy)
        hf = dict(regions=[(0.0, float(s.box[2]))], heatfinterval=1)
        o = oracle_mod.Oracle(s)
        o.set_hf(hf)
        o.mklist()
        want = o.calheatf()
        e = PgkEngine(s)
        e.set_hf(hf)
        e.mklist_cell()
        got = e.calheatf()
        assert np.abs(got - want).max() <= 1e-9 * np.abs(want).max(), (rr, dy)
        pot, pot_o = e.hf_atm()[0], o.hf_atm()[0]
        assert np.abs(pot - pot_o).max() <= 1e-9 * np.abs(pot_o).max(), (rr, dy)
        e.close()
