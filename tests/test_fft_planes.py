"""SPME convolution by whole planes (x lines and y pencils of a z plane in one
block) against the convolution pass by pass on the complex grid, and the
oracle: the three compiled sizes, other factors of 2, 3 and 5, grids that
differ by axis, the smallest, and planes that do not fit an SM (separate
passes).  Bars as tests/test_gpu_parity.py."""
import numpy as np
import pytest

from tests.conftest import rel_rms
from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(abi.PREC_FP64, 1e-10), (abi.PREC_MIXED, 1e-5)])
@pytest.mark.parametrize("nfft", [(8, 8, 8), (16, 16, 16), (32, 32, 32), (32, 32, 20), (64, 64, 24), (128, 128, 16),
                                  (30, 45, 25), (10, 50, 18), (48, 16, 150), (160, 180, 16)])
@pytest.mark.parametrize("tune", ["0", "1"])
def test_planes_match_passes(oracle_mod, monkeypatch, nfft, prec, tol, tune):
    from thrid_b200.pgk import PgkEngine
    s = S.small_box("propanol", nside=4, spacing=5.6)
    s.params.update(nfft1=nfft[0], nfft2=nfft[1], nfft3=nfft[2])
    monkeypatch.setenv("PGK_AUTOTUNE", tune)
    res = {}
    for r2c in ("1", "0"):
        monkeypatch.setenv("PGK_SPME_R2C", r2c)
        e = PgkEngine(s, dict(s.params, precision=prec))
        e.mklist_cell()
        res[r2c] = e.fft_pme()
        e.close()
    o = oracle_mod.Oracle(s)
    o.mklist()
    kf, ke, kv = o.fft_pmep()
    (f1, e1, v1), (f0, e0, v0) = res["1"], res["0"]
    assert rel_rms(f1, f0) < tol and rel_rms(f1, kf) < tol
    vt = np.abs(v0["pot_virit_coul"]).max()
    assert abs(e1["pot_ewk"] - e0["pot_ewk"]) < tol * abs(e0["pot_ewk"])
    assert np.abs(v1["pot_virit_coul"] - v0["pot_virit_coul"]).max() < tol * vt
