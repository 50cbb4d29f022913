"""Plain-mode systems of one context that run at the same time: from two threads,
and as chunks of a server's workers.  Each frame's terms run on side streams
that belong to its own call, so every row has the bits of a run alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rst():
    import rust_simulation_tools as r

    if r.device_count() < 1:
        pytest.skip("no GPU")
    return r


@pytest.fixture(scope="module")
def systems(rst, tmp_path_factory):
    from rust_simulation_tools import synthetic as S

    d, out = tmp_path_factory.mktemp("threads"), []
    for k, (n_rec, n_lig, frames) in enumerate([(150, 20, 24), (700, 30, 12), (90, 9, 24)]):
        s = S.make_system(n_rec, n_lig, seed=81 + k)
        fr = S.make_frames(s, frames, seed=91 + k)
        prm = str(d / ("%d.prmtop" % k))
        S.write_prmtop(s, prm)
        b = rst.BindingSystem(rst.read_prmtop(prm), s.receptor_residues, s.ligand_residues, mode="plain",
                              sa_params=rst.SaParams(n_sphere_points=240))
        out.append((b, fr, b.run(fr, decompose=True)))
    return out


def test_systems_in_threads(systems):
    got, errors = [[] for _ in systems], []
    start = threading.Barrier(len(systems))

    def work(k):
        try:
            b, fr, _ = systems[k]
            start.wait()
            for _ in range(6):
                got[k].append(b.run(fr, decompose=True))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(systems))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for (_, _, alone), runs in zip(systems, got):
        for e, dec in runs:
            np.testing.assert_array_equal(e, alone[0])
            np.testing.assert_array_equal(dec, alone[1])


def test_systems_in_a_server(rst, systems):
    srv = rst.Server(max_inflight=3)
    ids = [[srv.submit(b, fr) for _ in range(4)] for b, fr, _ in systems]
    for (_, _, alone), mine in zip(systems, ids):
        for i in mine:
            np.testing.assert_array_equal(srv.wait(i, 60000), alone[0])
    srv.close()
