"""Register-resident RATTLE (rigid water, stars of 2, 3 and 1 arms) against the
oracle's rattle_c / rattlep_v: near the constraint surface and far from it
(where the carried reciprocal is replaced by a division).  The sweeps are the
same, so the results agree to rounding: 1e-9 A, the trajectory bar of
tests/test_gpu_parity.py."""
import numpy as np
import pytest

from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "water": lambda: S.small_box("water", nside=4, spacing=3.1),           # 64 rigid groups
    "water_ragged": lambda: S.small_box("water", nside=3, spacing=3.1),    # 27
    "propanol": lambda: S.small_box("propanol", nside=4, spacing=5.6),     # CH3, CH2, OH
    "butane": lambda: S.small_box("butane", nside=4, spacing=5.4, nfft=24, order=5),
}


@pytest.mark.parametrize("amp", [0.002, 0.05, 0.2])
@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_matches_oracle(oracle_mod, name, amp):
    from thrid_b200.pgk import PgkEngine
    s = SYSTEMS[name]()
    rng = np.random.default_rng(9)
    old = s.atmcor.copy()
    x = old + rng.uniform(-amp, amp, old.shape)
    dt = S.fs_to_reduced(1.0)
    o = oracle_mod.Oracle(s)
    o.set_state(x, s.atmvel)
    o.rattle_c(old, 1e-7, dt)
    o.rattlep_v(1e-7)
    e = PgkEngine(s, dict(s.params, precision=abi.PREC_FP64))
    e.upload_state(x, s.atmvel)
    e.rattle_c(old, 1e-7, dt)
    e.rattlep_v(1e-7)
    xo, vo, _ = o.get_state()
    xg, vg, _ = e.download_state()
    assert np.abs(xg - xo).max() <= 1e-9
    assert np.abs(vg - vo).max() <= 1e-9 * max(1.0, np.abs(vo).max())


def test_no_convergence_is_reported():
    from thrid_b200.pgk import PgkEngine, PgkError
    s = SYSTEMS["water"]()
    x = s.atmcor.copy()
    x[0, 0] = np.nan
    e = PgkEngine(s, dict(s.params, precision=abi.PREC_FP64))
    e.upload_state(x, s.atmvel)
    with pytest.raises(PgkError) as err:
        e.rattle_c(s.atmcor, 1e-7, S.fs_to_reduced(1.0))
    assert err.value.status == abi.PGK_E_RATTLE_NOCONV
