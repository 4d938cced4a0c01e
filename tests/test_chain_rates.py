"""Nose-Hoover chain updates at rates on both sides of the series limit of the
chain's exponential (argument 1/16), against the oracle: the bars are those of
tests/test_gpu_parity.py (1e-9 A, 1e-8 relative to the largest velocity or
rate), because one step of the same formulas differs by rounding only."""
import numpy as np
import pytest

from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["nhc", "mtk"])
@pytest.mark.parametrize("x", [0.0, 0.03, 0.0625, -0.0624, 0.2, -0.2])
def test_one_step_matches_oracle(oracle_mod, kind, x):
    from thrid_b200.pgk import PgkEngine
    s = S.small_box("propanol", nside=4, spacing=5.6)
    dt = S.fs_to_reduced(1.0)
    md = abi.md_struct(dt, mchain=4, text=S.kelvin_to_reduced(300.0), tfreq=1.0e13 * S.TIMEREF,
                       vfreq=0.2e12 * S.TIMEREF, pext=S.pa_to_reduced(1.0e5), pcont_axis=abi.PCONT_ISO,
                       degfree=s.degfree_all, ifrattle=1, eps_rattle=1e-7)
    # the update's argument is yscoeff dt / next / 8 times the rate
    rate = x * 8.0 * md.next / (md.yscoeff[0] * dt)

    def chain():
        ch = abi.chain_init(s.box)
        ch.vlogs[3] = rate                 # the chain's end drives no other rate quadratically
        return ch

    o = oracle_mod.Oracle(s)
    o.set_chain(chain())
    status, _ = o.moldyn({"nhc": 1, "mtk": 2}[kind], 0, 1, md)
    assert status == 0
    e = PgkEngine(s, dict(s.params, precision=abi.PREC_FP64))
    e.set_chain(chain())
    getattr(e, "moldyn_" + kind)(0, 1, md)
    xo, vo, bo = o.get_state()
    xg, vg, bg = e.download_state()
    assert np.abs(xg - xo).max() <= 1e-9
    assert np.abs(vg - vo).max() <= 1e-8 * max(1.0, np.abs(vo).max())
    assert np.abs(np.array(bg) - np.array(bo)).max() <= 1e-12 * np.max(bo)
    oc, gc = o.get_chain(), e.get_chain()
    for name in ("xlogs", "vlogs"):
        a, b = np.array(getattr(gc, name)[:4]), np.array(getattr(oc, name)[:4])
        assert np.abs(a - b).max() <= 1e-8 * max(1.0, np.abs(b).max())
