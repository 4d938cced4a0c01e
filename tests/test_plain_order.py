"""The plain order of sums (pgk_ctx::plain_order) of heat-flux contexts and served
replicas, where a result amplifies the rounding of the positions: a bare 1/r
cut off at rrcut in the heat-flux records, hundreds of steps in a served run.

The numbers below were recorded from the engine with one row per lower cluster
and plain RATTLE sweeps.  Bars: a record's sums differ by FP32 rounding of their
terms, 1e-6 and below, and by 7e-4 when one pair is on the other side of the
cutoff; equal bits of every step's positions leave a served replica's velocities
equal, and another order of the sums moves these atoms by 7e-4 and 1e-3.  2e-5
lies between."""
import numpy as np
import pytest

from tests.conftest import rel_rms
from thrid_b200 import abi
from thrid_b200 import systems as S

pytestmark = pytest.mark.gpu

MD = dict(ifrattle=1, outinterval=0)

# 2,187 water atoms (seed 56), two regions, 14 records: kinetic transport, one
# potential and one virial column, the total
RECORD_COLS = (0, 7, 15, 17)
RECORDS = """
    -6.665135743e-03 4.922718237e-02 8.008143422e-02 1.473951234e-01 -2.632975630e-03 -8.087747706e-02 -1.256363616e-01 -2.451354061e-01
    -5.335791349e-03 3.211971094e-03 6.633789406e-02 8.510246348e-02 -6.153324035e-03 -3.907715186e-02 -8.489155732e-02 -1.605306385e-01
    -2.374081471e-03 -1.560215138e-02 4.458933204e-02 4.458694343e-02 -1.187368784e-02 -1.014244092e-02 -4.945327806e-02 -9.683880310e-02
    2.060901249e-03 -1.269061370e-01 -1.783155643e-02 -1.275729403e-01 -2.032901541e-02 7.806760410e-02 3.597648452e-02 7.370840137e-02
    7.616146746e-03 -1.408118368e-01 -1.819900336e-02 -1.394072806e-01 -3.197103921e-02 6.690287340e-02 1.269946765e-01 1.477972314e-01
    1.537307352e-02 -1.770328494e-01 -2.932325011e-02 -1.814024639e-01 -4.870570423e-02 1.076832123e-01 2.169399591e-01 2.670755419e-01
    2.305426820e-02 -2.026913098e-01 -6.585777978e-02 -2.379579839e-01 -6.893530574e-02 1.475524280e-01 3.001934503e-01 3.748358876e-01
    3.297888618e-02 -1.934616376e-01 -9.423143854e-02 -2.487972869e-01 -9.528134373e-02 2.195450012e-01 3.797737114e-01 5.042577929e-01
    3.936109935e-02 -1.283847360e-01 -8.076052669e-02 -1.649852091e-01 -1.216107621e-01 2.435204914e-01 4.553029817e-01 5.807083100e-01
    4.761615625e-02 -1.587753475e-01 -1.260524067e-01 -2.331461059e-01 -1.521024511e-01 3.043018058e-01 5.048892401e-01 6.629249052e-01
    4.261361182e-02 -1.385313540e-01 -1.577035765e-01 -2.498990427e-01 -1.694359137e-01 3.926297098e-01 5.225222882e-01 7.528742663e-01
    4.952038297e-02 -1.609098793e-01 -1.851049546e-01 -2.927891761e-01 -1.959373256e-01 4.205515866e-01 5.347238338e-01 7.668416197e-01
    5.331110808e-02 -1.894410778e-02 -2.403180414e-01 -2.019980487e-01 -2.138329157e-01 5.015621116e-01 5.262662550e-01 8.209592781e-01
    4.566907450e-02 1.757400277e-01 -2.129830240e-01 1.284264313e-02 -2.130175614e-01 5.597965526e-01 4.759108735e-01 8.283469993e-01
"""

# velocities of a few atoms of 1,500-atom propanol replicas after 300 steps: seed -> (atoms, values)
SERVED = {
    4: ((1271, 1269, 1270, 1263), """
    8.959459927e-01 2.215518318e-01 1.159930519e+00 1.936019255e-01 7.343358779e+00 8.135648712e-01
    4.618229493e-01 -4.567162841e-01 -4.371196175e+00 -3.273958214e-01 -5.766340549e-01 -6.903276886e-01
"""),
    6: ((659, 655, 656, 657, 658, 652), """
    -1.247076311e-02 1.044672059e-01 -1.041724595e+00 -2.329696806e+00 -7.682075020e-01 -1.365905831e+00
    -6.329759886e-01 -4.310347024e+00 -3.452165073e-01 1.494044796e+00 3.748795555e+00 -5.340401792e+00
    -1.274372458e+00 2.004780696e+00 -1.431964915e+00 3.107043534e+00 7.558237393e-01 1.057959919e+00
"""),
}


def _off(got, text):
    want = np.array(text.split(), dtype=float).reshape(got.shape)
    return np.linalg.norm(got - want) / np.linalg.norm(want)


def test_heat_flux_records_keep_their_values():
    from thrid_b200.pgk import PgkEngine
    s = S.small_box("water", nside=9, spacing=3.1, seed=56, precision=abi.PREC_MIXED, nfft=30, rcut=10.0)
    e = PgkEngine(s)
    lz = float(s.box[2])
    e.set_hf(dict(regions=[(0.0, 0.5 * lz), (0.5 * lz, lz)], heatfinterval=1))
    _, rec = e.moldyn_hf(0, 14, abi.md_struct(S.fs_to_reduced(1.0), **MD), cap=14)
    e.close()
    assert _off(rec[..., RECORD_COLS], RECORDS) < 2e-5


def test_served_replicas_keep_their_velocities():
    from thrid_b200.serve import ReplicaServer
    md = abi.md_struct(S.fs_to_reduced(1.0), **MD)
    srv = ReplicaServer(max_slots=2)
    ids = {k: srv.submit(S.small_box("propanol", nside=5, spacing=5.6, seed=k, precision=abi.PREC_MIXED, nfft=30, rcut=10.0),
                         md, kind=0, nsteps=300) for k in SERVED}
    got = {k: srv.result(i)[1] for k, i in ids.items()}
    srv.close()
    for k, (atoms, text) in SERVED.items():
        assert _off(got[k][list(atoms)], text) < 2e-5


@pytest.mark.parametrize("late", [False, True])
@pytest.mark.parametrize("name", ["water_1536", "propanol_8748", "butane_57400"])
def test_forces_of_plain_rows(oracle_mod, name, late):
    """Rows of the lower cluster, whole and sorted (several pieces in the 8,748-atom box of 27 cells), over a prune, a
    reuse and a prune again; late: the regions are set on a context that has segmented rows already."""
    from thrid_b200.pgk import PgkEngine
    s = {"water_1536": lambda: S.water_box(), "propanol_8748": lambda: S.propanol_box(nside=9, box=50.4),
         "butane_57400": lambda: S.butane_box(nmol=4100, nside=17, box=91.8)}[name]()
    o = oracle_mod.Oracle(s, threads=8)
    o.mklist()
    e = PgkEngine(s, dict(s.params, precision=abi.PREC_MIXED))
    hf = dict(regions=[(0.0, float(s.box[2]))], heatfinterval=1)
    x = s.atmcor.copy()
    if late:
        e.mklist_cell()
        e.ewaldr()
    e.set_hf(hf)
    if not late:
        e.mklist_cell()
    rng = np.random.default_rng(4)
    for amp in (0.0, 0.05, 0.3):
        x = x + rng.uniform(-amp, amp, x.shape) / np.sqrt(3.0)
        o.set_state(x)
        e.upload_state(x)
        want = o.ewaldrp()[0]
        assert rel_rms(e.ewaldr()[0], want) <= 1e-5
    e.close()
