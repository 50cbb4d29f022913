"""Launch shapes of the fused engine: what is reported is what runs, and a
frame's energies have the same bits on either side of each line that the number of frames draws."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rst():
    import rust_simulation_tools as r

    if r.device_count() < 1:
        pytest.skip("no GPU")
    return r


def system(rst, tmp_path, n_rec, n_lig, frames, **kw):
    from rust_simulation_tools import synthetic as S

    s = S.make_system(n_rec, n_lig, seed=17)
    fr = S.make_frames(s, frames, seed=18)
    prm = str(tmp_path / "s.prmtop")
    S.write_prmtop(s, prm)
    return rst.BindingSystem(rst.read_prmtop(prm), s.receptor_residues, s.ligand_residues, **kw), fr


@pytest.mark.parametrize("probe,warps", [(1.4, 4), (40.0, 2)])
def test_sasa_warps(rst, tmp_path, probe, warps):
    """A probe that makes every atom a neighbour of every other: four atoms' lists do not fit shared memory."""
    b, fr = system(rst, tmp_path, 1500, 20, 1, sa_params=rst.SaParams(probe_radius=probe, n_sphere_points=10))
    b.run(fr)
    assert b.tuning()["sasa_warps_per_block"] == warps


@pytest.mark.parametrize("n_rec,n_lig,frames", [(120, 12, (1, 12, 30)), (1000, 30, (1, 2, 3, 220))])
def test_bits_do_not_depend_on_the_number_of_frames(rst, tmp_path, n_rec, n_lig, frames):
    """Four, two and one warps an atom (2,368 and 1,184 atoms a batch), two and three pair blocks an SM (18,944 items)."""
    b, fr = system(rst, tmp_path, n_rec, n_lig, max(frames), sa_params=rst.SaParams(n_sphere_points=100))
    first, dec = b.run(fr[:1], decompose=True)
    for f in frames:
        e, d = b.run(fr[:f], decompose=True)
        np.testing.assert_array_equal(e[0], first[0])
        np.testing.assert_array_equal(d[0], dec[0])
