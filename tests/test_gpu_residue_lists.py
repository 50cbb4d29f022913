"""Residue lists that name a residue twice, or in both parts: the batched engine
evaluates the parts independently, as the single-frame call does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rst():
    import rust_simulation_tools as r

    if r.device_count() < 1:
        pytest.skip("no GPU")
    return r


@pytest.mark.parametrize("rec,lig", [([0, 0], [1]), ([0], [1, 1]), ([0, 1, 0], [2, 3]), ([0, 1], [1, 2]), ([0], [0]),
                                     ([3, 0, 1], [2])])
def test_repeated_residues(rst, rec, lig):
    rng = np.random.default_rng(4)
    n = 30
    top = rst.AmberTopology.from_arrays(rng.uniform(-5, 5, n), rng.choice([1.2, 1.5, 1.7], n), screen=[0.8] * n, n_types=2,
                                        atom_type_indices=rng.integers(0, 2, n), lj_acoef=[900.0, 700.0, 500.0],
                                        lj_bcoef=[8.0, 7.0, 6.0], nb_parm_index=[1, 2, 2, 3],
                                        residue_pointers=[0, 8, 15, 22])
    x = rng.uniform(0, 9.0, (2, n, 3)).astype(np.float32)
    sa = rst.SaParams(n_sphere_points=50)
    b = rst.BindingSystem(top, rec, lig, sa_params=sa)
    got, dec = b.run(x, decompose=True)
    assert dec.shape == (2, len(rec) + len(lig), 4)
    for f in range(2):
        nm = (x[f].astype(np.float64) * 0.1 * 10.0) / 10.0
        ref = rst.compute_binding_energy_single_frame(top, nm, rec, lig, sa_params=sa).as_array()
        ok = np.isfinite(ref)  # a part that holds an atom twice has pairs at distance zero
        assert (np.isfinite(got[f]) == ok).all()
        # the fused form's pair terms are FP32: 1e-6 of energies of up to 1e6 kcal/mol here
        np.testing.assert_allclose(got[f][ok], ref[ok], rtol=1e-6, atol=1e-6 * np.abs(ref[ok]).max())
