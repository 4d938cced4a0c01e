"""Admission of heat-flux replicas: the budget counts what a heat-flux context adds
to a plain one, with the estimate's margin of a quarter, so two replicas whose
sum is a byte over the budget do not run together."""
import pytest

from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu


def test_heat_flux_arrays_count_against_the_budget():
    from thrid_b200.serve import ReplicaServer, estimate_bytes
    s = S.small_box("water", nside=16, spacing=3.1, precision=abi.PREC_MIXED, nfft=45, rcut=9.0)
    hf = dict(regions=[(0.0, float(s.box[2]))], heatfinterval=1)
    cells = int(s.box[0] // s.params["rcut_book"]) ** 3
    slot = 8 + 4 + 32 + 16 + 64          # z, tag, velocities, region bits, pair sums
    atom = 8 * (8 + 24) + 24 + 3 * 4     # potentials, virials of one region, random forces, indices
    need = estimate_bytes(s) + 1.25 * (slot * (s.natom + 7 * cells) + atom * s.natom)
    md = abi.md_struct(S.fs_to_reduced(1.0), ifrattle=1, outinterval=0)
    srv = ReplicaServer(max_slots=2, hbm_budget_bytes=int(2 * need) - 1)
    ids = [srv.submit(s, md, kind=3, nsteps=6, hf=hf) for _ in range(2)]
    r = [srv.result(i) for i in ids]
    srv.close()
    assert r[1][5][1] >= r[0][5][2]      # the second starts after the first has finished
