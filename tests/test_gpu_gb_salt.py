"""Binding GB difference where burial changes the radii by angstroms and salt
screens strongly, so that exp(-0.73 kappa f) of complex and part are far apart:
the fused engine against the restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rst():
    import rust_simulation_tools as r

    if r.device_count() < 1:
        pytest.skip("no GPU")
    return r


@pytest.mark.parametrize("scale", [1.0, 1.3, 1.6])
@pytest.mark.parametrize("eps,salt", [(78.5, 0.0), (78.5, 0.15), (78.5, 1.0), (10.0, 1.0), (4.0, 5.0)])
def test_buried_ligand(rst, oracle, tmp_path, scale, eps, salt):
    from rust_simulation_tools import synthetic as S

    s = S.make_system(300, 200, seed=61)
    fr = (S.make_frames(s, 1, seed=62, sigma=0.05) * scale).astype(np.float32)
    fr[0, 300:] += (fr[0, :300].mean(0) - fr[0, 300:].mean(0)) * 0.8  # the ligand inside the receptor
    prm = str(tmp_path / "b.prmtop")
    S.write_prmtop(s, prm)
    kw = dict(solvent_dielectric=eps)
    got = rst.BindingSystem(rst.read_prmtop(prm), s.receptor_residues, s.ligand_residues,
                            gb_params=rst.GbParams(model=2, salt_concentration=salt, **kw),
                            sa_params=rst.SaParams(n_sphere_points=20)).run(fr)[0]
    ref = oracle.binding_frame(oracle.Topology.load(prm), (fr[0].astype(np.float64) * 0.1) * 10.0, s.receptor_residues,
                               s.ligand_residues, gb=oracle.gb_params("obc2", salt=salt, **kw), sa=oracle.sa_params(n_points=20),
                               accurate=True)
    # 1e5 pairs of up to 60 kcal/mol, each to a few FP32 roundings (and a difference to 1e-6 of itself)
    for k, name in ((1, "complex_polar"), (4, "receptor_polar"), (7, "ligand_polar"), (10, "delta_polar")):
        assert abs(got[k] - ref[name]) <= np.sqrt(1e5) * 60 * 3e-7, (name, got[k], ref[name])
