"""Row segments and pruned rows of the pair kernel, both precisions: boxes whose
clusters are split over 8, a few or one segment per row, evaluated at the
start (prune), after a small move (pruned rows reused) and after a large one
(pruned again), against the oracle on the same pair list.  Bars as
tests/test_gpu_parity.py: FP64 1e-12 (the same formulas; 1/r, the spline index
and the image by other roundings, a few ulp), mixed 1e-5."""
import numpy as np
import pytest

from tests.conftest import rel_rms
from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu

CASES = {
    "propanol_324": lambda: S.small_box("propanol", nside=3, spacing=5.6),        # 41 clusters
    "water_1536": lambda: S.water_box(),                                          # 2^3 cells
    "propanol_8748": lambda: S.propanol_box(nside=9, box=50.4),                   # 2-3 segments
    "butane_38416": lambda: S.butane_box(nmol=2744, nside=14, box=75.6),          # one segment
    "butane_57400": lambda: S.butane_box(nmol=4100, nside=17, box=91.8),          # cluster frame, ragged count
}


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("name", sorted(CASES))
def test_forces_across_prunes(oracle_mod, name, prec):
    from thrid_b200.pgk import PgkEngine
    s = CASES[name]()
    o = oracle_mod.Oracle(s, threads=8)
    o.mklist()
    e = PgkEngine(s, dict(s.params, precision=prec))
    e.mklist_cell()
    rng = np.random.default_rng(4)
    x = s.atmcor.copy()
    for amp in (0.0, 0.05, 0.3):
        x = x + rng.uniform(-amp, amp, x.shape) / np.sqrt(3.0)
        o.set_state(x)
        e.upload_state(x)
        want, we, wv = o.ewaldrp()
        got, ge, gv = e.ewaldr()
        assert rel_rms(got, want) <= (1e-12 if prec == abi.PREC_FP64 else 1e-5)
        tol = 1e-10 if prec == abi.PREC_FP64 else 1e-5
        for k in ("pot_vdw", "pot_elc"):
            assert abs(ge[k] - we[k]) <= tol * max(1.0, abs(we[k]))
        for k in ("pot_virit_coul", "pot_virit_lj"):
            assert np.abs(gv[k] - wv[k]).max() <= tol * max(1.0, np.abs(wv[k]).max())


@pytest.mark.parametrize("name", ["water_1536", "butane_57400"])
def test_fp64_barostat_tensor_matches_the_split_one(name):
    """The combined-tensor mode (anisotropic MTK steps) against the split tensors' sum: one MTK step each way."""
    from thrid_b200.pgk import PgkEngine
    s = CASES[name]()
    ends = []
    for interval in (1, 1 << 30):          # energies every step (split tensors) / never (combined)
        md = abi.md_struct(S.fs_to_reduced(1.0), mchain=3, text=S.kelvin_to_reduced(250.0), tfreq=1e13 * S.TIMEREF,
                           vfreq=0.2e12 * S.TIMEREF, pext=S.pa_to_reduced(1e5), pcont_axis=abi.PCONT_ANISO,
                           degfree=s.degfree_all, outinterval=interval)
        e = PgkEngine(s, dict(s.params, precision=abi.PREC_FP64))
        e.set_chain(abi.chain_init(s.box))
        e.moldyn_mtk(0, 2, md)
        ch = e.get_chain()
        ends.append(np.array(list(ch.vboxg)))
    assert np.abs(ends[0] - ends[1]).max() <= 1e-10 * np.abs(ends[0]).max()
