"""awsem_profile_step: a time for every kernel of a step, none for the pair
list's decision, which is part of the prepare kernel."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_a_time_for_every_kernel(prec, tmp_path, gpu_lib):
    from awsemmd_b200 import engine, synth

    ff = synth.forcefield_dir(str(tmp_path / "ff"))
    with engine.AwsemBatch.from_arrays(ff, [synth.chain_arrays(60, 41)], precision=prec) as s:
        s.run(1)
        ms = s.profile_step(3)
    assert len(ms) == engine.NKERNELS
    assert ms.pop("nl_decide") == 0.0
    assert all(t > 0.0 for t in ms.values())
