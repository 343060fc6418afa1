"""Force calls that a handle evaluates from its recorded graph: the bits of a
fresh handle's directly queued call, forces and energies, whatever the order of
term groups, and after a pair-list overflow met by a recorded call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RECORDED = 12  # calls with one set of terms, enough for its graph


def _equal(a, b):
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_term_groups_in_turn(prec, tmp_path, gpu_lib):
    from awsemmd_b200 import engine, synth

    c = synth.chain_arrays(70, 6400, n_mem_per_window=4)
    ff = synth.forcefield_dir(str(tmp_path / "ff"))
    x0 = c["x"].reshape(-1, 3)
    x1 = x0 + np.random.default_rng(6).normal(0.0, 0.05, x0.shape)
    want = {}
    for t in range(1, 8):
        with engine.AwsemBatch.from_arrays(ff, [c], precision=prec) as fresh:
            want[t] = fresh.compute(x1, terms=t)
    with engine.AwsemBatch.from_arrays(ff, [c], precision=prec) as s:
        for k in range(RECORDED):
            for t in range(1, 8):
                s.compute(x0, terms=t)
        for t in (7, 1, 1, 2, 4, 7, 3, 5, 6, 7):
            _equal(s.compute(x1, terms=t), want[t])


def test_pair_list_overflow(tmp_path, gpu_lib):
    from awsemmd_b200 import synth
    from awsemmd_b200.engine import AwsemSystem

    files = synth.write_system(synth.config_system(1), str(tmp_path / "c1"))
    with AwsemSystem(files, precision="mixed") as fresh:
        x0, _ = fresh.get_state()
        squeezed = x0.mean(axis=0) + 0.2 * (x0 - x0.mean(axis=0))
        want, tight = fresh.compute(x0), fresh.compute(squeezed)
    with AwsemSystem(files, precision="mixed") as s:
        for k in range(RECORDED):
            _equal(s.compute(x0), want)
        _equal(s.compute(squeezed), tight)  # the list grows, the recording goes, the call is evaluated again
        for k in range(RECORDED):
            _equal(s.compute(x0), want)
        _equal(s.compute(squeezed), tight)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_short_windows(prec, tmp_path, gpu_lib):
    """A run in windows of seven steps, single steps at first and graphs of
    five later, has the bits of the run in one call."""
    from awsemmd_b200 import engine, synth

    c = synth.chain_arrays(35, 6600, n_mem_per_window=2)
    ff = synth.forcefield_dir(str(tmp_path / "ff"))
    kw = dict(t_start=330.0, t_stop=290.0, seed=5)
    n, part = 490, 7
    with engine.AwsemBatch.from_arrays(ff, [c], precision=prec) as s:
        s.run_window(n, (0, n), False, **kw)
        want = (*s.get_state(0), s.forces(0), s.energies(0))
    with engine.AwsemBatch.from_arrays(ff, [c], precision=prec) as s:
        for at in range(0, n, part):
            s.run_window(part, (0, n), at > 0, **kw)
        got = (*s.get_state(0), s.forces(0), s.energies(0))
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
