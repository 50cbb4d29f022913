"""Single-term functions at the limits of their inputs: coincident atoms whose
intrinsic radius is zero, coordinates at infinity without a cutoff."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rst():
    import rust_simulation_tools as r

    if r.device_count() < 1:
        pytest.skip("no GPU")
    return r


def pair(rst, oracle, radii, screen, x, **kw):
    arrays = dict(screen=screen, residue_pointers=[0])
    q = [3.0, -2.0, 1.0]
    nm = np.array(x) / 10.0
    e = rst.compute_gb_energy(rst.AmberTopology.from_arrays(q, radii, **arrays), nm, rst.GbParams(**kw))
    ref = oracle.gb_energy(oracle.Topology.from_arrays(q, radii, **arrays), nm * 10.0,
                           oracle.gb_params(("hct", "obc1", "obc2")[kw["model"]], salt=kw["salt_concentration"],
                                            cutoff=kw["cutoff"]))
    return e.total, e.born_radii(), ref[0], ref[1]


@pytest.mark.parametrize("model", [0, 1, 2])
@pytest.mark.parametrize("radii,screen", [([0.09, 0.09, 1.5], [0.0, 0.0, 0.8]), ([0.09, 1.5, 1.2], [0.8, 0.0, 0.8]),
                                          ([1.5, 1.5, 1.2], [0.8, 0.7, 0.8])])
def test_coincident_atoms(rst, oracle, model, radii, screen):
    x = [[0.0, 0.0, 0.0], [0.0, 0.0, 0.0], [3.0, 0.0, 0.0]]
    _, R, _, oR = pair(rst, oracle, radii, screen, x, model=model, salt_concentration=0.0, cutoff=9999.0)
    np.testing.assert_allclose(R, oR, rtol=1e-12)


@pytest.mark.parametrize("model", [0, 1, 2])
def test_radii_of_an_infinite_distance(rst, oracle, model):
    x = [[0.0, 0.0, 0.0], [2.0, 0.0, 0.0], [0.0, np.inf, 0.0]]
    e, R, oe, oR = pair(rst, oracle, [1.5, 1.7, 1.2], [0.8, 0.7, 0.8], x, model=model, salt_concentration=0.0, cutoff=np.inf)
    np.testing.assert_allclose(R, oR, rtol=1e-12)
    np.testing.assert_allclose(e, oe, rtol=1e-12)


@pytest.mark.parametrize("model", [0, 1, 2])
def test_salt_at_an_infinite_distance(rst, oracle, model):
    x = [[0.0, 0.0, 0.0], [2.0, 0.0, 0.0], [0.0, np.inf, 0.0]]
    e, _, oe, _ = pair(rst, oracle, [1.5, 1.7, 1.2], [0.8, 0.7, 0.8], x, model=model, salt_concentration=0.15, cutoff=np.inf)
    np.testing.assert_allclose(e, oe, rtol=1e-12)


def test_binding_difference_with_an_atom_at_infinity(rst, tmp_path):
    """Receptor x ligand GB pairs vanish with the distance: infinity is as good as 1e12 A."""
    from rust_simulation_tools import synthetic as S

    s = S.make_system(60, 9, seed=5)
    fr = np.repeat(S.make_frames(s, 1, seed=6, sigma=0.05) * 1.6, 2, axis=0).astype(np.float32)
    fr[0, 7, 1], fr[1, 7, 1] = 1e12, np.inf
    prm = str(tmp_path / "i.prmtop")
    S.write_prmtop(s, prm)
    b = rst.BindingSystem(rst.read_prmtop(prm), s.receptor_residues, s.ligand_residues, sa_params=rst.SaParams(n_sphere_points=20),
                          gb_params=rst.GbParams(salt_concentration=0.15, cutoff=np.inf))
    e = np.concatenate([b.run(fr[k:k + 1]) for k in range(2)])
    np.testing.assert_allclose(e[1, 10], e[0, 10], rtol=1e-9)  # qq / (eps 1e12 A) of a hundred pairs


@pytest.mark.parametrize("probe", [-0.5, -1.6, -3.0, -4.0])
def test_sasa_with_a_negative_probe(rst, oracle, probe):
    """Expanded radii below zero: points on a sphere of their size, tested against spheres of theirs."""
    rng = np.random.default_rng(9)
    n = 60
    nm = rng.uniform(0, 0.8, (n, 3))
    radii = rng.choice([1.2, 1.5, 1.7, 1.8], n)
    arrays = dict(screen=[0.8] * n, residue_pointers=[0])
    s = rst.compute_sa_energy(rst.AmberTopology.from_arrays(np.zeros(n), radii, **arrays), nm,
                              rst.SaParams(probe_radius=probe, n_sphere_points=70))
    ref = oracle.sa_energy(oracle.Topology.from_arrays(np.zeros(n), radii, **arrays), nm * 10.0,
                           oracle.sa_params(probe=probe, n_points=70))[2]
    np.testing.assert_array_equal(s.per_atom_sasa(), ref)


def test_atom_types_without_tables(rst):
    """A topology with atom types but no number of types has no Lennard-Jones terms."""
    rng = np.random.default_rng(2)
    n = 40
    x = rng.uniform(0, 1.5, (n, 3))
    kw = dict(screen=[0.8] * n, residue_pointers=[0, 30], n_types=0, lj_acoef=(), lj_bcoef=(), nb_parm_index=())
    q, radii = rng.uniform(-5, 5, n), [1.5] * n
    a, b = (rst.AmberTopology.from_arrays(q, radii, atom_type_indices=t, **kw) for t in (np.zeros(n), np.arange(n) * 1000))
    assert rst.compute_mm_energy(b, x).vdw == rst.compute_mm_energy(a, x).vdw == 0.0
    fr = (x[None] * 10.0).astype(np.float32)
    ea, eb = (rst.BindingSystem(t, [0], [1], sa_params=rst.SaParams(n_sphere_points=20)).run(fr) for t in (a, b))
    np.testing.assert_array_equal(ea, eb)
