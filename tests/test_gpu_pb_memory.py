"""Device memory of a plain PB energy with focusing: a coarse grid too large for
the two solves of the pair to run side by side is solved for one after the
other, however small the fine grid is."""
import gc
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rst():
    import rust_simulation_tools as r

    if r.device_count() < 1:
        pytest.skip("no GPU")
    return r


def test_large_coarse_grid(rst):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(4)
    n, span = 30, 6.0
    x = rng.uniform(0, span, (n, 3))
    x[0], x[1] = 0.0, span
    top = rst.AmberTopology.from_arrays(rng.uniform(-9, 9, n), rng.choice([1.2, 1.5, 1.7], n), screen=[0.8] * n)
    p = rst.PbParams(grid_spacing=0.5, grid_buffer=3.0, fillratio=40.0, fscale=2, max_iterations=60)
    coarse = (int(np.ceil(span * 40.0)) + 1) ** 3  # points at 1 A
    rst.compute_pb_energy(top, x / 10.0, rst.PbParams(grid_spacing=0.5, grid_buffer=3.0, fillratio=0.0))
    gc.collect()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    least, stop = [free], threading.Event()

    def sample():
        while not stop.is_set():
            least[0] = min(least[0], torch.cuda.mem_get_info()[0])
            time.sleep(2e-4)

    t = threading.Thread(target=sample)
    t.start()
    e = rst.compute_pb_energy(top, x / 10.0, p)
    stop.set()
    t.join()
    assert np.isfinite(e.total) and max(e.diag["dims"]) < 30
    # a solve: four maps, its potential, three arrays of levels and a code (65 bytes a point); beside it the charges and
    # the other side's potential (16); up to 256 MB (19) of it may come from what the library keeps between calls
    used = free - least[0]
    assert 40 * coarse < used < 100 * coarse, used / coarse
