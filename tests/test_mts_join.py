"""Multiple time steps with SPME and the bonded terms in the short group and the
pairs in the long one: the long evaluation begins where the short one's streams
join.  Captured steps, eager steps, one stream and three give the same mixed-
precision bits (integer force sums)."""
import numpy as np
import pytest

from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["nve", "mtk"])
def test_short_spme_long_pairs(monkeypatch, kind):
    from thrid_b200.pgk import PgkEngine
    s = S.small_box("propanol", nside=5, spacing=5.6, seed=3, precision=abi.PREC_MIXED, nfft=30, rcut=10.0)
    short = {k: abi.MTS_SHORT for k in ("mts_ewk", "mts_bond", "mts_angl", "mts_tors", "mts_torsrb")}
    md = abi.md_struct(S.fs_to_reduced(1.0), nstep_short=2, mchain=3, text=S.kelvin_to_reduced(300.0), tfreq=1e13 * S.TIMEREF,
                       vfreq=0.2e12 * S.TIMEREF, pext=S.pa_to_reduced(1e5), pcont_axis=abi.PCONT_ANISO,
                       degfree=s.degfree_all, ifrattle=1, outinterval=0)
    got = []
    for graphs, streams in (("0", "1"), ("0", "3"), ("1", "3")):
        monkeypatch.setenv("PGK_GRAPHS", graphs)
        monkeypatch.setenv("PGK_STREAMS", streams)
        e = PgkEngine(s, dict(s.params, **short))
        e.set_chain(abi.chain_init(s.box))
        (e.moldyn_nve if kind == "nve" else e.moldyn_mtk)(0, 30, md)
        x, v, box = e.download_state()
        e.close()
        got.append((x, v, box))
    for other in got[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(got[0], other))
