"""A finite cutoff belongs to the GB terms: Lennard-Jones and Coulomb energies of
the fused engine do not change with it, in tiles inside, across and beyond it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rst():
    import rust_simulation_tools as r

    if r.device_count() < 1:
        pytest.skip("no GPU")
    return r


@pytest.mark.parametrize("n_rec,n_lig", [(33, 31), (127, 1), (129, 127), (700, 64)])
@pytest.mark.parametrize("salt", [0.0, 0.15])
@pytest.mark.parametrize("cutoff", [2.0, 9.0, 20.0])
def test_mm_has_no_cutoff(rst, oracle, tmp_path, n_rec, n_lig, salt, cutoff):
    from rust_simulation_tools import synthetic as S

    s = S.make_system(n_rec, n_lig, seed=100 + n_rec)
    fr = (S.make_frames(s, 1, seed=3, sigma=0.05) * 1.6).astype(np.float32)
    prm = str(tmp_path / "c.prmtop")
    S.write_prmtop(s, prm)
    top = rst.read_prmtop(prm)
    got, far = (rst.BindingSystem(top, s.receptor_residues, s.ligand_residues, sa_params=rst.SaParams(n_sphere_points=20),
                                  gb_params=rst.GbParams(salt_concentration=salt, cutoff=c)).run(fr)[0]
                for c in (cutoff, 9999.0))
    ref = oracle.binding_frame(oracle.Topology.load(prm), (fr[0].astype(np.float64) * 0.1) * 10.0, s.receptor_residues,
                               s.ligand_residues, gb=oracle.gb_params("obc2", salt=salt, cutoff=cutoff),
                               sa=oracle.sa_params(n_points=20), accurate=True)
    # pair terms in FP32, sums of 32 of them: rounding relative to the terms' size, as without a cutoff
    for k, name in ((0, "complex_mm"), (3, "receptor_mm"), (6, "ligand_mm"), (9, "delta_mm")):
        tol = 1e-3 if k == 9 else 1e-6 * max(abs(ref[name]), 1e2)
        assert abs(got[k] - ref[name]) <= tol, (name, got[k], ref[name])
        assert abs(got[k] - far[k]) <= tol, (name, got[k], far[k])
