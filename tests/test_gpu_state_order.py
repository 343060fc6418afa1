"""State moved in and out of replicas whose atoms change order on the host or
on the device, around the sizes where the way changes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_round_trip(tmp_path, gpu_lib):
    from awsemmd_b200 import engine, synth

    def many(n):  # n residues, in chains of at most 500
        if n <= 500:
            return synth.chain_arrays(n, 6300 + n, n_mem_per_window=1)
        k = -(-n // 500)
        return synth.packed_arrays([n // k + (j < n % k) for j in range(k)], 500.0, 6300 + n, n_mem_per_window=1)

    sizes = (2, 555, 556, 3000, 3001)
    ff = synth.forcefield_dir(str(tmp_path / "ff"))
    rng = np.random.default_rng(8)
    with engine.AwsemBatch.from_arrays(ff, [many(n) for n in sizes]) as b:
        want = []
        for k, n in enumerate(sizes):
            x, v = rng.normal(size=(3 * n, 3)), rng.normal(size=(3 * n, 3))
            b.set_state(x, rng.normal(size=(3 * n, 3)), k)
            b.set_state(v=v, r=k)
            want.append((x, v))
        for k, (x, v) in enumerate(want):
            gx, gv = b.get_state(k)
            assert np.array_equal(gx, x) and np.array_equal(gv, v), sizes[k]
        ax, av = b.get_state_all()
        assert np.array_equal(ax, np.concatenate([w[0] for w in want]))
        assert np.array_equal(av, np.concatenate([w[1] for w in want]))
        b.set_state_all(av, ax)
        for k, (x, v) in enumerate(want):
            gx, gv = b.get_state(k)
            assert np.array_equal(gx, v) and np.array_equal(gv, x), sizes[k]
