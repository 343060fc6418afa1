"""The forms the engine picks by size give the same bits: small chains alone
(residue terms by tasks, detection on the whole pair list) and beside enough
residues for the other forms (a thread per residue, the near list)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = (2, 5, 31, 32, 33, 65)  # around a warp of residues, and the shortest chains


@pytest.fixture(scope="module")
def chains():
    from awsemmd_b200 import synth

    return ([synth.chain_arrays(n, 5100 + n, n_mem_per_window=3) for n in LENGTHS],
            synth.chain_arrays(500, 5600, n_mem_per_window=1))


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_forms_agree(prec, chains, tmp_path, gpu_lib):
    from awsemmd_b200 import engine, synth

    small, filler = chains
    ff = synth.forcefield_dir(str(tmp_path / "ff"))
    kw = dict(t_start=350.0, t_stop=300.0)
    got = []
    for desc in (small, small + [filler] * 140):
        with engine.AwsemBatch.from_arrays(ff, desc, precision=prec, seeds=list(range(1, len(desc) + 1))) as b:
            b.run(12, **kw)
            got.append([(*b.get_state(k), b.forces(k), b.energies(k)) for k in range(len(small))])
    for k, (a, b) in enumerate(zip(*got)):
        for u, v in zip(a[:3], b[:3]):
            assert np.array_equal(u, v), LENGTHS[k]
        np.testing.assert_allclose(b[3], a[3], rtol=1e-12, atol=1e-9)
