"""radm2_rosenbrock_host begins behind what is already on the context's stream: uploads, copies of
the state and transposes enqueued just before it neither disturb it nor are disturbed."""
import numpy as np
import pytest

import radm2b200
from conftest import ATOL, RTOL
from radm2b200 import inputs

pytestmark = pytest.mark.gpu
N = 100003
PERS, WIDE = radm2b200.SCHED_PERSISTENT, radm2b200.lib.PLACE_LU_TMEM_WIDE


def host_call(s, cells, nchunk):
    y = np.ascontiguousarray(cells["VAR"]).copy()
    ipar, rpar = radm2b200.default_params(hstart=6.0)
    assert s.rosenbrock_host(y, cells["FIX"], cells["TEMP"], cells["RC_N2O5"], cells["JV"], 0.0, 60.0, ATOL, RTOL, rpar, ipar,
                             nchunk=nchunk) == 1
    return y, list(ipar[10:17])


@pytest.mark.parametrize("opts,nchunk", [(dict(), 8), (dict(), 1), (dict(schedule=PERS, block_threads=128), 4)])
def test_host_call_waits_for_earlier_work(opts, nchunk):
    torch = pytest.importorskip("torch")
    a, b = inputs.make_cells(N, 3, "plain", 0.3), inputs.make_cells(N, 4, "mixed", 0.4)
    with radm2b200.Solver(**opts) as s:
        want = host_call(s, b, nchunk)
    pinned = {k: torch.from_numpy(np.ascontiguousarray(a[k])).pin_memory().numpy() for k in ("VAR", "FIX", "TEMP", "RC_N2O5", "JV")}
    out = torch.empty((40, 59, N), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with radm2b200.Solver(**opts) as s:
        host_call(s, a, nchunk)  # allocates the staging buffer
        for _ in range(3):
            s.set_cells(pinned)
            for k in range(len(out)):
                s.get_state_device(out[k].data_ptr(), N)
            got = host_call(s, b, nchunk)
            assert np.array_equal(got[0], want[0]) and got[1] == want[1]
            s.synchronize()
            assert bool((out == torch.from_numpy(np.ascontiguousarray(a["VAR"].T)).cuda()).all())


def test_host_call_leaves_the_visiting_order():
    """A cell order set by the caller holds for later calls, and the chunks do without it."""
    cells = inputs.make_cells(5000, 6, "mixed", 0.4)
    order = np.random.RandomState(2).permutation(5000).astype(np.int32)
    with radm2b200.Solver(schedule=PERS, placement=WIDE) as s:
        want = host_call(s, cells, 5)
        s.set_cell_order(order)
        got = host_call(s, cells, 5)
    assert np.array_equal(got[0], want[0]) and got[1] == want[1]


def test_device_bytes_count_the_second_stream():
    """The second compute stream's scratch is the context's: radm2_device_bytes grows by what the
    device loses."""
    torch = pytest.importorskip("torch")
    cells = inputs.make_cells(20000, 8, "plain", 0.3)
    with radm2b200.Solver() as s:
        host_call(s, cells, 1)
        held, free = s.device_bytes(), torch.cuda.mem_get_info()[0]
        host_call(s, cells, 8)
        grown, lost = s.device_bytes() - held, free - torch.cuda.mem_get_info()[0]
        assert grown > 32 << 20 and abs(lost - grown) <= 8 << 20  # allocations come in pages of 2 MiB
        host_call(s, cells, 8)
        assert s.device_bytes() - held == grown
