"""Positions that are not finite, or finite and absurdly far out, in a force
call or a run: the call reports the former, and the next call with ordinary
positions has a fresh handle's bits, on a pair list of its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _equal(a, b):
    for u, v in zip(a, b):
        assert np.array_equal(u, v)


# one chain scanned directly, and enough residues for a cell grid; directly queued calls and recorded ones
@pytest.mark.parametrize("calls", [1, 12])
@pytest.mark.parametrize("chains", [1, 5])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_next_call_is_clean(prec, chains, calls, tmp_path, gpu_lib):
    from awsemmd_b200 import engine, synth

    length = 40 if chains == 1 else 430
    c = synth.packed_arrays([length] * chains, 60.0 if chains == 1 else 250.0, 65, n_mem_per_window=2)
    ff = synth.forcefield_dir(str(tmp_path / "ff"))
    x = c["x"].reshape(-1, 3)
    with engine.AwsemBatch.from_arrays(ff, [c], precision=prec) as fresh:
        want = fresh.compute(x)
    with engine.AwsemBatch.from_arrays(ff, [c], precision=prec) as s:
        for k in range(calls):
            _equal(s.compute(x), want)
        # the contact bead, the oxygen, the whole residue
        for atoms in (slice(17, 18), slice(16, 17), slice(15, 18)):
            for value in (np.nan, np.inf, -np.inf):
                bad = x.copy()
                bad[atoms, 2] = value
                f = np.full_like(x, 0.25)
                with pytest.raises(engine.AwsemError, match="non-finite"):
                    s.compute(bad, f=f)
                assert (f == 0.25).all()
                _equal(s.compute(x), want)
            for value in (1e12, -1e30):
                far = x.copy()
                far[atoms, 2] = value
                s.compute(far)
                _equal(s.compute(x), want)
        bad = x.copy()
        bad[17, 2] = np.inf
        s.set_state(x=bad)
        with pytest.raises(engine.AwsemError, match="non-finite"):
            s.run(3, dt=1.0, langevin=False)
        _equal(s.compute(x), want)
