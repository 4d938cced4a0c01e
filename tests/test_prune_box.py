"""Pruned rows under a changing box: the box shrinks between two evaluations on one
pair list, with the positions kept, scaled along, or scaled and moved, by less
than what forces a new prune of pairs inside the box.  Pairs across a face come
closer by up to the whole change of the box.  Against the same evaluation
without pruned rows (PGK_PRUNE_BUFFER=0).  Bars: FP64 1e-12 (equal terms in
another order), mixed 1e-5, as tests/test_pair_segments.py; a pair missed near
the cutoff is above 1e-4."""
import numpy as np
import pytest

from tests.conftest import rel_rms
from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(abi.PREC_FP64, 1e-12), (abi.PREC_MIXED, 1e-5)])
@pytest.mark.parametrize("move", ["box", "scaled", "scaled_moved", "one_axis"])
@pytest.mark.parametrize("nside", [10, 14])
def test_no_pair_is_missed_when_the_box_shrinks(monkeypatch, prec, tol, move, nside):
    from thrid_b200.pgk import PgkEngine
    s = S.small_box("water", nside=nside, spacing=6.4, nfft=16, rcut=12.0)    # far apart: no overlap across a face
    shrink = np.array([1.0, 1.0, 0.98]) if move == "one_axis" else np.full(3, 0.98)
    x1 = s.atmcor.copy()
    x2 = x1 * (shrink if move.startswith("scaled") else 1.0)
    if move == "scaled_moved":
        x2 = x2 + np.random.default_rng(2).uniform(-0.1, 0.1, x2.shape)
    got = {}
    for buf in ("0.7", "0"):
        monkeypatch.setenv("PGK_PRUNE_BUFFER", buf)
        e = PgkEngine(s, dict(s.params, precision=prec))
        e.upload_state(x1)
        e.mklist_cell()
        e.ewaldr()                                    # prunes
        e.upload_state(x2, None, s.box * shrink)
        got[buf] = e.ewaldr()[0]
        e.close()
    assert rel_rms(got["0.7"], got["0"]) <= tol
