"""RATTLE of a star whose first bond has turned by exactly 90 degrees at its length:
R.r_old = 0 while that constraint is satisfied (the reference skips it), and
not zero once the second bond's correction has moved the centre.  Against the
oracle, bar as tests/test_rattle_forms.py."""
import numpy as np
import pytest

from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
def test_a_bond_turned_by_90_degrees(oracle_mod, prec):
    from thrid_b200.pgk import PgkEngine
    s = S.small_box("propanol", nside=4, spacing=5.6)
    old = s.atmcor.copy()
    arms = {}
    for k, (c, h) in enumerate(s.const_ij):
        arms.setdefault(int(c), []).append((int(h), float(s.const_d[k])))
    stars = {c: a for c, a in arms.items() if len(a) == 2}
    assert len(stars) == 2 * s.nmole      # the CH2 stars
    x = old.copy()
    for c, ((h1, d1), (h2, d2)) in stars.items():
        old[h1] = old[c] + [d1, 0.0, 0.0]
        old[h2] = old[c] + [d2, 0.0, 0.0]
        x[h1] = old[c] + [0.0, d1, 0.0]
        x[h2] = old[c] + [1.03 * d2, 0.0, 0.0]
    dt = S.fs_to_reduced(1.0)
    o = oracle_mod.Oracle(s)
    o.set_state(x, s.atmvel)
    o.rattle_c(old, 1e-7, dt)
    e = PgkEngine(s, dict(s.params, precision=prec))
    e.upload_state(x, s.atmvel)
    e.rattle_c(old, 1e-7, dt)
    xo, vo, _ = o.get_state()
    xg, vg, _ = e.download_state()
    assert np.isfinite(xo).all()
    assert np.abs(xg - xo).max() <= 1e-9
    assert np.abs(vg - vo).max() <= 1e-9 * max(1.0, np.abs(vo).max())
