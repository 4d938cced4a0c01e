"""Region sums of the heat-flux record (k_flux_*) against the oracle's per-atom
arrays summed by calheatf, where the forms of the regions and atoms matter:
more regions than one walk of a row takes, gaps and overlaps, slabs outside
the box, planes exactly on atoms, molecule-based and atom-based z, pairs inside
one molecule.  Bars as tests/test_hf.py: FP64 sums of the same FP64 terms in
another order (1e-9 of the largest entry), FP32 pair terms 2e-4."""
import numpy as np
import pytest

from tests.test_hf import HF_FP64, HF_MIXED, _gpu_engine, small_slab
from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu


def _regions(kind, s):
    lz = float(s.box[2])
    if kind == "one":
        return [(0.0, lz)]
    if kind == "narrow":
        w = lz / 32
        return [(k * w, (k + 1) * w) for k in range(32)]
    if kind == "ragged":      # gap, overlap, slab beyond the box, descending order
        return [(0.6 * lz, 0.9 * lz), (0.3 * lz, 0.65 * lz), (-5.0, 0.2 * lz), (0.95 * lz, lz + 7.0), (0.31 * lz, 0.32 * lz)]
    z = np.sort(s.atmcor[:, 2] - lz * np.floor(s.atmcor[:, 2] / lz))
    n = len(z)
    return [(z[n // 7], z[n // 2]), (z[n // 2], z[3 * n // 4]), (z[3 * n // 4], z[-1])]   # planes on atoms


def _system(what):
    if what == "slab":
        return small_slab()
    s = S.small_box("butane", nside=4, spacing=5.4, nfft=24, order=5)
    s.regions = dict(hf=dict(regions=[], heatfinterval=1))
    return s


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("what,kind", [("slab", "one"), ("slab", "narrow"), ("slab", "ragged"), ("slab", "planes"),
                                       ("butane", "one"), ("butane", "narrow"), ("butane", "planes")])
def test_record_matches_oracle(oracle_mod, what, kind, prec):
    s = _system(what)
    hf = dict(s.regions["hf"], regions=_regions(kind, s), langevin=[])
    o = oracle_mod.Oracle(s)
    o.set_hf(hf)
    o.mklist()
    want = o.calheatf()
    e = _gpu_engine(s, prec)
    e.set_hf(hf)
    e.mklist_cell()
    got = e.calheatf()
    bar = HF_FP64 if prec == abi.PREC_FP64 else HF_MIXED
    assert np.abs(got - want).max() <= bar * np.abs(want).max()
    again = e.calheatf()      # the sums were left zero
    assert np.abs(again - got).max() <= 1e-9 * np.abs(want).max()


@pytest.mark.parametrize("interval,end", [(1, 3), (2, 4), (3, 6)])
def test_arrays_hold_the_last_evaluation_of_a_run(oracle_mod, interval, end):
    s = small_slab()
    hf = dict(s.regions["hf"], heatfinterval=interval)
    md = abi.md_struct(S.fs_to_reduced(1.0), ifrattle=1, outinterval=0)
    o = oracle_mod.Oracle(s)
    o.set_hf(hf)
    _, _, want = o.moldyn_hf(0, end, md)
    e = _gpu_engine(s, abi.PREC_FP64)
    e.set_hf(hf)
    _, got = e.moldyn_hf(0, end, md)
    assert got.shape == want.shape
    assert np.abs(got - want).max() <= 1e-7 * np.abs(want).max()
    for a, b in zip(e.hf_atm(), o.hf_atm()):
        assert np.abs(a - b).max() <= 1e-7 * np.abs(b).max()
