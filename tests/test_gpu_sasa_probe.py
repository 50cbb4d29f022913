"""SASA of the fused engine with large probes, where an FP32 point test errs by
more than it does at 1.4 A: pairs whose nearest sphere point lies on the other
atom's expanded sphere to 1e-7 A, against the restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rst():
    import rust_simulation_tools as r

    if r.device_count() < 1:
        pytest.skip("no GPU")
    return r


@pytest.mark.parametrize("probe", [1.4, 10.0, 25.0, 60.0])
def test_points_on_a_sphere(rst, oracle, probe):
    rng = np.random.default_rng(3)
    wrong = 0
    for _ in range(40):
        # two sphere points: the one at +y faces the other atom
        ri = round(float(rng.uniform(1.2, 1.8)), 3)
        fr = np.zeros((1, 2, 3), np.float32)
        fr[0, 1, 1] = np.float32(ri + 2 * probe + rng.uniform(1.2, 1.8))
        x = (fr[0].astype(np.float64) * 0.1) * 10.0
        rj = (x[1, 1] - (ri + probe)) - probe + float(rng.choice([-1, 1]) * 10 ** rng.uniform(-9, -6))
        arrays = dict(screen=[0.8, 0.8], residue_pointers=[0, 1])
        top = rst.AmberTopology.from_arrays([1.0, -1.0], [ri, rj], **arrays)
        otop = oracle.Topology.from_arrays([1.0, -1.0], [ri, rj], **arrays)
        got = rst.BindingSystem(top, [0], [1], sa_params=rst.SaParams(probe_radius=probe, n_sphere_points=2)).run(fr)[0]
        ref = oracle.binding_frame(otop, x, [0], [1], sa=oracle.sa_params(probe=probe, n_points=2), accurate=True)
        # whole points: half a sphere of area each
        wrong += abs(got[2] - ref["complex_sa"]) > 1e-9 * abs(ref["complex_sa"])
    assert wrong == 0
