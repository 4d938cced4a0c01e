"""ewaldkp_hf on half the wave set, in runs and groups of four waves: the
smallest sets (3 waves held), runs that leave remainders, one and several
segments, atom counts around a block of 256.  Bar as tests/test_ewk_hf.py:
FP64 sums in another order, 1e-10 of the largest entry."""
import numpy as np
import pytest

from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.mark.parametrize("nside,kmax", [(3, 1), (3, 2), (4, 3), (5, 6), (7, 9)])     # 81, 192, 375, 1029 atoms
@pytest.mark.parametrize("netq", [0, 1])
def test_matches_oracle(oracle_mod, nside, kmax, netq):
    from thrid_b200.pgk import PgkEngine
    s = S.small_box("water", nside=nside, spacing=3.1, rcut=nside * 3.1 / 2 - 2.2)
    s.params["ifnetqcorrp"] = netq
    if netq:
        s.atmchrg = s.atmchrg + 0.01 * abs(s.atmchrg).max()
    want = oracle_mod.Oracle(s).ewaldkp_hf(kmax)
    got = PgkEngine(s, dict(s.params, precision=abi.PREC_FP64)).ewaldkp_hf(kmax)
    assert got["nwave"] == want["nwave"]
    for k in ("force", "pot_atm", "viri_atm", "pot_virit_coul"):
        assert np.abs(got[k] - want[k]).max() <= TOL * np.abs(want[k]).max()
    for k in ("pot_ewk", "pot_ewk_cc"):
        assert abs(got[k] - want[k]) <= TOL * max(abs(want[k]), 1e-300)
