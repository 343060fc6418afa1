"""A handle records its force call in a graph at the third call: later calls at
other positions, steps and term groups give a fresh handle's bits; state moved
in and out between runs comes back as it was put."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [2, 33, 90])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_force_calls(prec, length, tmp_path, gpu_lib):
    from awsemmd_b200 import engine, synth

    c = synth.chain_arrays(length, 6100 + length, n_mem_per_window=4)
    ff = synth.forcefield_dir(str(tmp_path / "ff"))
    x0 = c["x"].reshape(-1, 3)
    rng = np.random.default_rng(5)
    xs = [x0 + rng.normal(0.0, 0.05, x0.shape) for _ in range(6)]
    # groups as a host with and without its own pair style asks for them; a change starts the recording again
    terms = [7, 7, 7, 7, 7, 7, 1, 1, 1, 1, 7, 2, 2, 2, 2]
    with engine.AwsemBatch.from_arrays(ff, [c], precision=prec) as s:
        for k, t in enumerate(terms):
            if k == 5:
                s.set_launch_shapes((1, 37, 5, 0))  # drops the recorded call
            x = xs[k % 6] if k != 12 else xs[0] + 30.0  # far enough to rebuild the pair list
            f0 = np.full_like(x, 0.25)
            f, e = s.compute(x, step=k, terms=t, f=f0.copy())
            assert s.step == k
            with engine.AwsemBatch.from_arrays(ff, [c], precision=prec) as fresh:
                fw, ew = fresh.compute(x, step=k, terms=t, f=f0.copy())
                assert np.array_equal(f, fw), (k, t)
                np.testing.assert_allclose(e, ew, rtol=1e-12, atol=1e-9)
                assert np.array_equal(s.forces(), fresh.forces())


def test_state_round_trip(tmp_path, gpu_lib):
    from awsemmd_b200 import engine, synth

    cs = [synth.chain_arrays(n, 6200 + n, n_mem_per_window=1) for n in (7, 40, 33)]
    ff = synth.forcefield_dir(str(tmp_path / "ff"))
    with engine.AwsemBatch.from_arrays(ff, cs) as b:
        rng = np.random.default_rng(7)
        want = []
        for k, c in enumerate(cs):
            x, v = rng.normal(size=(3 * c["n_res"], 3)), rng.normal(size=(3 * c["n_res"], 3))
            b.set_state(x=x, r=k)
            b.set_state(v=v, r=k)
            want.append((x, v))
        for k, (x, v) in enumerate(want):
            gx, gv = b.get_state(k)
            assert np.array_equal(gx, x) and np.array_equal(gv, v)
        ax, av = b.get_state_all()
        assert np.array_equal(ax, np.concatenate([w[0] for w in want]))
        assert np.array_equal(av, np.concatenate([w[1] for w in want]))
