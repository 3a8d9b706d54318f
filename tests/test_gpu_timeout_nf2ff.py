"""Reading the NF2FF accumulators into no buffer waits for the steps before it
and reports a bounded device wait that ran out (efs_debug_set_wait, as in
test_gpu_timeout.py: nothing faults or hangs, the waits give up by design)."""
import pytest

from test_gpu_parity import nf2ff_inputs, rand_coeffs

pytestmark = pytest.mark.gpu
EFS_ERR_TIMEOUT = 5


def test_reading_into_no_buffer_reports_the_wait(cuda_engine_cls):
    N = (20, 18, 24)
    g = cuda_engine_cls()
    assert g.initGPU()
    g.init(N, rand_coeffs(N, 50))
    nf = nf2ff_inputs(N, nfreq=2, inset=4)
    g.configureNF2FFAccumulation(nf)
    n = 2 * 6 * nf["numPoints"]
    g.debugSetWait(2_000_000, skip_plane=5)
    g.iterate(1)
    assert g._lib.efs_read_nf2ff(g._h, None, None, n) == EFS_ERR_TIMEOUT
    assert g._lib.efs_read_nf2ff(g._h, None, None, n) == 0      # reported once and cleared
    g.debugSetWait()
    g.destroy()
