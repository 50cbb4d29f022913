"""Batched PB in a server: the chains of grids that run beside a solve's own
stream have the priority of the chunk's rank."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rst():
    import rust_simulation_tools as r

    if r.device_count() < 1:
        pytest.skip("no GPU")
    return r


def priorities(b):
    from rust_simulation_tools import _native as N

    st = np.zeros(8)
    assert N.lib.rstg_system_pb_stats(b._h, st.ctypes.data_as(C.POINTER(C.c_double))) == 0
    return tuple(st[6:])


def test_chains_have_the_chunk_s_priority(rst, tmp_path):
    from rust_simulation_tools import synthetic as S

    s = S.make_system(90, 9, seed=55)
    fr = S.make_frames(s, 2, seed=56)
    prm = str(tmp_path / "p.prmtop")
    S.write_prmtop(s, prm)
    b = rst.BindingSystem(rst.read_prmtop(prm), s.receptor_residues, s.ligand_residues,
                          pb_params=rst.PbParams(grid_spacing=0.8, grid_buffer=4.0, fillratio=0.0))
    alone = b.run(fr)
    assert priorities(b) == (0.0, 0.0)
    srv = rst.Server(max_inflight=2)  # two levels; a request by itself is the oldest and takes the higher one
    np.testing.assert_array_equal(srv.wait(srv.submit(b, fr), 60000), alone)
    mine, chains = priorities(b)
    assert mine < 0.0 and chains == mine
    srv.close()
    np.testing.assert_array_equal(b.run(fr), alone)  # and back on the context's stream
    assert priorities(b) == (0.0, 0.0)
