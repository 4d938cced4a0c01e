"""Per-atom heat-flux arrays (k_hf_pair) against the oracle's, where the rows
and regions take its different ways: one region, more regions than one walk
takes, planes exactly on atoms, and molecules so large that most pairs of a
row lie inside one.  Bars as tests/test_hf.py."""
import numpy as np
import pytest

from tests.test_flux_sums import _regions
from tests.test_hf import HF_FP64, HF_MIXED, _gpu_engine, small_slab
from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu


def _system(what):
    if what == "slab":
        return small_slab()
    s = S.small_box("butane", nside=4, spacing=5.4, nfft=24, order=5)
    s.regions = dict(hf=dict(regions=[], heatfinterval=1))
    n = len(s.molept_list)
    if what == "one molecule":
        s.molept_index = np.array([0, n], s.molept_index.dtype)
    if what == "two molecules":          # rows of both classes
        s.molept_index = np.array([0, n // 2, n], s.molept_index.dtype)
    return s


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("what,kind", [("slab", "one"), ("slab", "narrow"), ("slab", "planes"), ("butane", "ragged"),
                                       ("one molecule", "one"), ("one molecule", "narrow"),
                                       ("two molecules", "ragged"), ("two molecules", "planes")])
def test_arrays_match_oracle(oracle_mod, what, kind, prec):
    s = _system(what)
    hf = dict(s.regions["hf"], regions=_regions(kind, s), langevin=[])
    o = oracle_mod.Oracle(s)
    o.set_hf(hf)
    o.mklist()
    o.calheatf()
    pw, Ww = o.hf_atm()
    e = _gpu_engine(s, prec)
    e.set_hf(hf)
    e.mklist_cell()
    e.calheatf()
    pg, Wg = e.hf_atm()
    bar = HF_FP64 if prec == abi.PREC_FP64 else HF_MIXED
    assert pg.shape == pw.shape and Wg.shape == Ww.shape
    assert np.abs(pg - pw).max() <= bar * np.abs(pw).max()
    assert np.abs(Wg - Ww).max() <= bar * np.abs(Ww).max()
