"""SPME by whole planes and by separate passes rounds alike: the choice between
them is a measured time, and the mixed engine's results are the same bits from
run to run.  Grids whose axes the separate passes compile and the planes do not
(one compiled length beside another one), compiled pairs, and grids without a
compiled length.  The FP64 engine spreads with FP64 atomics, so its bits are
not compared."""
import numpy as np
import pytest

from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nfft", [(64, 48, 20), (48, 64, 16), (128, 64, 12), (64, 128, 16), (32, 64, 18), (128, 96, 10),
                                  (36, 128, 12), (64, 64, 24), (128, 128, 16), (48, 48, 48), (30, 45, 25)])
def test_planes_and_passes_give_the_same_bits(monkeypatch, nfft):
    from thrid_b200.pgk import PgkEngine
    s = S.small_box("propanol", nside=4, spacing=5.6)
    s.params.update(nfft1=nfft[0], nfft2=nfft[1], nfft3=nfft[2])
    got = {}
    for plane in ("0", "1"):
        monkeypatch.setenv("PGK_FFT_PLANE", plane)
        e = PgkEngine(s, dict(s.params, precision=abi.PREC_MIXED))
        e.mklist_cell()
        got[plane] = e.fft_pme()
        e.close()
    (f0, e0, v0), (f1, e1, v1) = got["0"], got["1"]
    assert np.array_equal(f0, f1)
    assert e0["pot_ewk"] == e1["pot_ewk"]
    assert np.array_equal(v0["pot_virit_coul"], v1["pot_virit_coul"])
