"""FP32 partial sums of the descreening integral: over 64 or 128 columns, as
systems have had them since their launch shapes were timed (the values below
are of that build), whatever the shape that runs now."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rst():
    import rust_simulation_tools as r

    if r.device_count() < 1:
        pytest.skip("no GPU")
    return r


# (receptor atoms, ligand atoms, frames, autotune): polar energies (complex, receptor, ligand, difference) of two frames
KNOWN = {
    (800, 40, 3, True): [[-19759.341305064714, -18682.44094411991, -1177.7168995679456, 100.816086836895],
                         [-19814.8786398025, -18733.102772652448, -1183.3132735460615, 101.53736841422747]],
    (800, 40, 3, False): [[-19759.341270101486, -18682.440939776534, -1177.716899444578, 100.81608682274937],
                          [-19814.878643716627, -18733.10276815658, -1183.3132753140187, 101.53736843809526]],
    (420, 40, 2, True): [[-10302.883668101927, -9391.487021717781, -873.9988700024278, -37.397550382227855],
                         [-10277.45409130422, -9396.913973216417, -842.4925206961609, -38.047683609641346]],
    (2000, 30, 3, True): [[-52421.41282909917, -52078.099226445884, -346.12052984276863, 2.806564719720635],
                          [-52492.1902878899, -52146.46829870027, -348.5421477816998, 2.820374470733375]],
}


@pytest.mark.parametrize("n_rec,n_lig,frames,autotune", KNOWN)
def test_partial_sums(rst, tmp_path, n_rec, n_lig, frames, autotune):
    from rust_simulation_tools import synthetic as S

    s = S.make_system(n_rec, n_lig, seed=61)
    fr = (S.make_frames(s, frames, seed=62, sigma=0.05) * 1.6).astype(np.float32)
    prm = str(tmp_path / "s.prmtop")
    S.write_prmtop(s, prm)
    b = rst.BindingSystem(rst.read_prmtop(prm), s.receptor_residues, s.ligand_residues, autotune=autotune,
                          gb_params=rst.GbParams(model=2, solvent_dielectric=78.5, salt_concentration=0.15),
                          sa_params=rst.SaParams(n_sphere_points=97 + (not autotune)))
    got = b.run(fr)
    ref = np.array(KNOWN[n_rec, n_lig, frames, autotune])
    # the same FP32 sums, added in another order in FP64 (some 1e5 terms, differences of 1e4 kcal/mol): 64 columns
    # against 128 are 1e-9 to 1e-8 of these energies apart
    assert np.abs(got[:2, [1, 4, 7, 10]] - ref).max() <= 1e-14 * np.sqrt(1e5) * np.abs(ref).max()
    again = b.run(fr[:1])  # the choice stays with the sizes, not with the number of frames
    np.testing.assert_array_equal(again[0], got[0])
