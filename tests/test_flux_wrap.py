"""Heat-flux records of molecules that lie several boxes away (a call before any
transcor has brought them back): calheatf shifts an atom's z, and a centre of
mass once more, by one box length and no more, so which region an atom's own
energy belongs to depends on the number of shifts.  Atom-based, molecule-based
and mixed typing against the oracle, all-pair lists, bar as tests/test_flux_sums.py."""
import numpy as np
import pytest

from tests.test_hf import HF_FP64
from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("typing", ["atom", "mole", "mixed"])
@pytest.mark.parametrize("kind,nside,spacing,rcut", [("propanol", 2, 6.2, 2.2), ("water", 3, 4.0, 3.0), ("butane", 2, 7.0, 2.5)])
def test_shifted_molecules(oracle_mod, kind, nside, spacing, rcut, typing):
    from thrid_b200.pgk import PgkEngine
    s = S.small_box(kind, nside=nside, spacing=spacing, seed=5, rcut=rcut)
    rng = np.random.default_rng(8)
    s.atmvel[:] = rng.normal(size=s.atmvel.shape) * np.sqrt(S.kelvin_to_reduced(200.0) / s.atmmass)[:, None]
    mol = np.empty(s.natom, dtype=int)
    mol[s.molept_list] = np.repeat(np.arange(s.nmole), np.diff(s.molept_index))
    s.atmcor[:] = s.atmcor + (rng.integers(-3, 4, (s.nmole, 3)) * s.box)[mol]
    by_mole = {"atom": 0 * mol, "mole": 0 * mol + 1, "mixed": mol % 2}[typing]
    lz = float(s.box[2])
    hf = dict(regions=[(k * lz / 3, (k + 1) * lz / 3) for k in range(3)], heatfinterval=1, hftyp=(1 + by_mole).astype(np.int32))
    o = oracle_mod.Oracle(s)
    o.set_hf(hf)
    o.mklist()
    want = o.calheatf()
    e = PgkEngine(s, dict(s.params, precision=abi.PREC_FP64))
    e.mklist_cell()
    e.set_hf(hf)
    got = e.calheatf()
    assert np.abs(got - want).max() <= HF_FP64 * np.abs(want).max()
    e.close()
