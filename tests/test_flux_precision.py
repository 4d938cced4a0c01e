"""Rounding error of mixed-precision heat-flux records: RMS over regions and 24
boxes of the difference to the FP64 engine at the same fixed-point positions, as
a share of the largest region's value.  The bars are the errors that FP32 pair
terms (correctly rounded 1/r, 1/r^2) summed in FP64 with FP64 velocities have,
recorded to three digits from an engine that forms the records from per-atom
FP64 virials, times 1.1; velocities and f . v in FP32 are 1.2 to 1.5 times
above them.  Columns of bare 1/r between molecules are left out: a pair that the
two precisions put on either side of the cutoff decides them."""
import numpy as np
import pytest

from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu

ERRORS = {   # kind, sites per side, spacing -> {record column: error}
    ("water", 9, 3.1): {8: 4.82e-7, 16: 4.64e-7},
    ("propanol", 6, 5.6): {5: 9.08e-8, 6: 7.54e-7, 8: 3.47e-7, 13: 2.02e-7, 14: 9.00e-7, 15: 4.79e-7, 16: 4.49e-7},
}


@pytest.mark.parametrize("box", sorted(ERRORS))
def test_records_are_as_exact_as_fp64_sums_of_fp32_pairs(box):
    from thrid_b200.pgk import PgkEngine
    kind, nside, spacing = box
    off = {c: [] for c in ERRORS[box]}
    for seed in range(24):
        s = S.small_box(kind, nside=nside, spacing=spacing, seed=seed, nfft=30, rcut=10.0)
        L = float(s.box[0])
        x = np.rint(s.atmcor / (L / 2.0 ** 32)) * (L / 2.0 ** 32)      # on the mixed engine's grid
        v = np.random.default_rng(seed).normal(size=x.shape) * np.sqrt(S.kelvin_to_reduced(300.0) / s.atmmass)[:, None]
        rec = {}
        for prec in (abi.PREC_FP64, abi.PREC_MIXED):
            e = PgkEngine(s, dict(s.params, precision=prec))
            e.set_hf(dict(regions=[(k * L / 5, (k + 1) * L / 5) for k in range(5)], heatfinterval=1))
            e.upload_state(x, v, s.box)
            e.mklist_cell()
            rec[prec] = e.calheatf()
            e.close()
        d = rec[abi.PREC_MIXED] - rec[abi.PREC_FP64]
        for c in off:
            off[c].append(np.sqrt(np.mean(d[:, c] ** 2)) / np.abs(rec[abi.PREC_FP64][:, c]).max())
    for c, bar in ERRORS[box].items():
        assert np.sqrt(np.mean(np.square(off[c]))) <= 1.1 * bar, c
